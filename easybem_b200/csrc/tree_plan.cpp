#include "tree_plan.h"

#include <algorithm>
#include <cmath>
#include <functional>
#include <utility>

namespace eb {

namespace {

struct Node {
  int lo, hi;      // cells
  int left, right; // children (-1: a cell)
  int parent;
  int height;      // 0 for a cell
};

// A small ball around the balls of cells [lo, hi): the centre of their box,
// moved towards the farthest ball.
dq ball_of(const std::vector<dq>& cell, int lo, int hi)
{
  d3 a = mk3(1e300, 1e300, 1e300), b = mk3(-1e300, -1e300, -1e300);
  for (int c = lo; c < hi; c++) {
    const dq& q = cell[c];
    a = mk3(std::min(a.x, q.x - q.w), std::min(a.y, q.y - q.w), std::min(a.z, q.z - q.w));
    b = mk3(std::max(b.x, q.x + q.w), std::max(b.y, q.y + q.w), std::max(b.z, q.z + q.w));
  }
  d3 m = 0.5 * (a + b);
  dq best{0.0, 0.0, 0.0, -1.0};
  for (int it = 0; it <= 6; it++) {
    double r = -1.0;
    d3 far = m;
    for (int c = lo; c < hi; c++) {
      const d3 v = mk3(cell[c].x, cell[c].y, cell[c].z) - m;
      const double d = std::sqrt(dot3(v, v)) + cell[c].w;
      if (d > r) {
        r = d;
        far = mk3(cell[c].x, cell[c].y, cell[c].z);
      }
    }
    if (best.w < 0.0 || r < best.w) best = dq{m.x, m.y, m.z, r};
    m = m + (1.0 / (it + 4.0)) * (far - m);
  }
  best.w *= 1.0 + 1e-12;
  return best;
}

// True when the centre of node k keeps kTreeMinStep of its radius from those of
// node j and its descendants.
bool clear_of(const std::vector<Node>& nodes, const std::vector<dq>& ball, int k, int j)
{
  const dq &x = ball[k], &y = ball[j];
  const d3 v = mk3(x.x - y.x, x.y - y.y, x.z - y.z);
  const double s = kTreeMinStep * x.w;
  if (dot3(v, v) < s * s) return false;
  return nodes[j].left < 0 || (clear_of(nodes, ball, k, nodes[j].left) && clear_of(nodes, ball, k, nodes[j].right));
}

// Pairs (c, j) as rows c of ascending j.
struct Rows {
  std::vector<int> ptr, col;
  Rows(int n, const std::vector<std::pair<int, int>>& pairs, bool both) : ptr(n + 1, 0)
  {
    for (const auto& q : pairs) {
      ptr[q.first + 1]++;
      if (both) ptr[q.second + 1]++;
    }
    for (int k = 0; k < n; k++) ptr[k + 1] += ptr[k];
    std::vector<int> fill(ptr.begin(), ptr.end() - 1);
    col.resize(ptr[n]);
    for (const auto& q : pairs) {
      col[fill[q.first]++] = q.second;
      if (both) col[fill[q.second]++] = q.first;
    }
    for (int k = 0; k < n; k++) std::sort(col.begin() + ptr[k], col.begin() + ptr[k + 1]);
  }
};

// How a list of pairs is cut into tasks, and the slots of a cell's forward sums.
struct Tasks {
  int chunk, log_parts = 0;
  explicit Tasks(int pairs) : chunk(std::min(kTreeNearChunk, std::max(1, pairs / kTreeNearTasks)))
  {
    while ((1 << log_parts) < kTreeNearParts && (pairs << log_parts) < kTreeNearTasks) log_parts++;
  }
  int parts() const { return 1 << log_parts; }  // above 1 with chunk 1 only
  int slots(int close) const { return (close + chunk) / chunk * parts(); }  // with the cell itself
};

int count_forward_slots(const TreePlan& plan)
{
  std::vector<int> close(plan.ncells, 0);
  for (const auto& q : plan.near) {
    close[q.first]++;
    close[q.second]++;
  }
  const Tasks cut(plan.ncells + 2 * (int)plan.near.size());
  int n = plan.all_close ? 0 : plan.ncells;  // the far slots
  for (int c : close) n += cut.slots(c);
  return n;
}

}  // namespace

void make_near_lists(const TreePlan& plan, bool both, TreeNear* out)
{
  // transposed slots first, then one forward slot per task, then the far slot
  const int nc = plan.ncells;
  const Rows close(nc, plan.near, !both);
  const Tasks cut(nc + (int)close.col.size());
  const int parts = cut.parts(), log_parts = cut.log_parts, chunk = cut.chunk;
  const int far_slots = plan.all_close ? 0 : 1;
  std::vector<int> trans(nc, 0);
  if (both)
    for (int j : close.col) trans[j]++;
  out->slot_off.assign(nc + 1, 0);
  for (int c = 0; c < nc; c++)
    out->slot_off[c + 1] =
        out->slot_off[c] + trans[c] + cut.slots(close.ptr[c + 1] - close.ptr[c]) + far_slots;
  std::vector<int> next(out->slot_off.begin(), out->slot_off.end() - 1);
  out->entries.reserve((close.col.size() + nc) * parts);
  for (int c = 0; c < nc; c++) {
    const int e0 = (int)out->entries.size();
    auto add = [&](int cell, int slot) {
      for (int part = 0; part < parts; part++)
        out->entries.push_back(make_int2(cell | part << kTreePartShift | log_parts << kTreePartsShift, slot));
    };
    add(c, -1);
    for (int q = close.ptr[c]; q < close.ptr[c + 1]; q++) add(close.col[q], both ? next[close.col[q]]++ : -1);
    const int e1 = (int)out->entries.size();
    int slot = out->slot_off[c] + trans[c];
    for (int e = e0; e < e1; e += chunk)
      out->tasks.push_back(make_int4(c, e, std::min(e1, e + chunk), slot++));
  }
  // the larger tasks first
  std::stable_sort(out->tasks.begin(), out->tasks.end(),
                   [](const int4& a, const int4& b) { return a.z - a.y > b.z - b.y; });
}

bool make_tree_plan(const HostMesh& h, TreePlan* plan)
{
  TreePlan& p = *plan;
  const int nc = h.ncells;
  p.ncells = nc;
  auto all_close = [&] {
    p.all_close = true;
    p.near.clear();
    for (int c = 0; c < nc; c++)
      for (int j = c + 1; j < nc; j++) p.near.push_back({c, j});
    make_near_lists(p, true, &p.sym);
    p.forward_slots = count_forward_slots(p);
    return true;
  };
  if (nc < kTreeMinCells) return all_close();
  std::vector<Node> nodes(nc);
  for (int c = 0; c < nc; c++) nodes[c] = Node{c, c + 1, -1, -1, -1, 0};
  std::function<int(int, int)> build = [&](int lo, int hi) {
    if (hi - lo == 1) return lo;
    const int mid = lo + split_cells(hi - lo);
    const int l = build(lo, mid), r = build(mid, hi);
    const int k = (int)nodes.size();
    nodes.push_back(Node{lo, hi, l, r, -1, 1 + std::max(nodes[l].height, nodes[r].height)});
    nodes[l].parent = nodes[r].parent = k;
    return k;
  };
  const int root = build(0, nc);
  if (nodes[root].height > kTreePasses * kTreeLevelsPerPass || (int)nodes.size() >= kTreeMaxNodes) return false;
  const int nn = p.nnodes = (int)nodes.size();
  for (int k = nc; k < nn; k++) p.child.push_back(make_int2(nodes[k].left, nodes[k].right));
  p.ball.resize(nn);
  for (int c = 0; c < nc; c++) {
    const double* b = &h.cell_ball[4 * (size_t)c];
    p.ball[c] = dq{b[0], b[1], b[2], std::max(h.cell_rho[c], 1e-3 * b[3])};
  }
  // a move scales with the inverse distance of the two centres, so an inner
  // node's centre keeps away from those of its descendants (symmetric meshes
  // put them at the same point)
  for (int k = nc; k < nn; k++) {
    const dq b = ball_of(p.ball, nodes[k].lo, nodes[k].hi);
    p.ball[k] = b;
    for (int t = 1; t < 64 && !(clear_of(nodes, p.ball, k, nodes[k].left) && clear_of(nodes, p.ball, k, nodes[k].right)); t++) {
      const double a = 2.4 * t, z = std::cos(1.7 * t), r = std::sqrt(1.0 - z * z), s = 0.004 * t * b.w;
      p.ball[k] = dq{b.x + s * r * std::cos(a), b.y + s * r * std::sin(a), b.z + s * z, b.w + s};
    }
  }

  // the tree against itself
  struct Far {
    int a, b;
    unsigned key;  // 255 - f: sorts the pairs that need most degrees first
  };
  std::vector<Far> far;
  far.reserve(32 * (size_t)nc);
  std::vector<std::pair<int, int>> near;  // close cells, the earlier one first
  near.reserve(20 * (size_t)nc);
  const double share = nc > kTreeSmallCells ? kTreeMaxShare : kTreeSmallShare;
  const long long limit = std::min((long long)(0.5 * share * nc * nc), (long long)(kTreeMaxSlotBytes / (kCell * sizeof(double))));
  std::vector<std::pair<int, int>> stack(1, {root, root});
  while (!stack.empty()) {
    const auto [a, b] = stack.back();
    stack.pop_back();
    const Node &A = nodes[a], &B = nodes[b];
    if (a == b) {
      if (A.left < 0) continue;
      stack.push_back({A.left, A.right});
      stack.push_back({A.left, A.left});
      stack.push_back({A.right, A.right});
      continue;
    }
    const dq &x = p.ball[a], &y = p.ball[b];
    const d3 d = mk3(x.x - y.x, x.y - y.y, x.z - y.z);
    const double d2 = dot3(d, d);
    if (separated(x.w, y.w, d2, kTreeRatio)) {
      far.push_back({a, b, 255u - degree_share(x.w, y.w, d2, kTreeRatio)});
    } else if (A.left < 0 && B.left < 0) {
      near.push_back({std::min(a, b), std::max(a, b)});
      if ((long long)near.size() > limit) return nc <= kTreeAllCloseCells && all_close();
    } else if (B.left < 0 || (A.left >= 0 && x.w >= y.w)) {
      stack.push_back({A.left, b});
      stack.push_back({A.right, b});
    } else {
      stack.push_back({a, B.left});
      stack.push_back({a, B.right});
    }
  }

  // separated pairs in both directions, by target, each list sorted by
  // (255 - f, source)
  std::vector<int> count(nn + 1, 0);
  for (const Far& f : far) {
    count[f.a + 1]++;
    count[f.b + 1]++;
  }
  for (int k = 0; k < nn; k++) count[k + 1] += count[k];
  std::vector<int> fill(count.begin(), count.end() - 1);
  std::vector<unsigned> src(2 * far.size());
  std::vector<char> used(nn, 0);  // its multipole is read
  for (const Far& f : far) {
    src[fill[f.a]++] = f.key << 24 | (unsigned)f.b;
    src[fill[f.b]++] = f.key << 24 | (unsigned)f.a;
    used[f.a] = used[f.b] = 1;
  }
  p.has_local.assign(nn, 0);
  // targets with the longest lists first (the last wave then holds short ones)
  std::vector<int> order;
  for (int k = 0; k < nn; k++)
    if (count[k + 1] > count[k]) {
      order.push_back(k);
      p.has_local[k] = 1;
    }
  std::stable_sort(order.begin(), order.end(),
                   [&](int a, int b) { return count[a + 1] - count[a] > count[b + 1] - count[b]; });
  p.m2l.src.reserve(src.size());
  for (int k : order) {
    std::sort(src.begin() + count[k], src.begin() + count[k + 1]);
    p.m2l.tgt.push_back(k);
    for (int q = count[k]; q < count[k + 1]; q++) p.m2l.src.push_back((int)((255u - (src[q] >> 24)) << 24 | (src[q] & 0xffffffu)));
    p.m2l.ptr.push_back((int)p.m2l.src.size());
  }

  // upward: pass s forms the nodes of heights (s L, (s + 1) L] from their
  // descendants of height at most s L (the topmost on each path)
  std::vector<int> byheight;
  for (int k = nc; k < nn; k++) byheight.push_back(k);
  std::stable_sort(byheight.begin(), byheight.end(), [&](int a, int b) { return nodes[a].height > nodes[b].height; });
  std::vector<std::vector<int>> sources(nn);
  for (int k : byheight) {  // from the top: a used node makes its sources used
    if (!used[k]) continue;
    const int base = (nodes[k].height - 1) / kTreeLevelsPerPass * kTreeLevelsPerPass;
    std::function<void(int)> gather = [&](int j) {
      if (nodes[j].height <= base) {
        sources[k].push_back(j);
        used[j] = 1;
        return;
      }
      gather(nodes[j].left);
      gather(nodes[j].right);
    };
    gather(k);
  }
  for (int k = nc; k < nn; k++) {
    if (!used[k]) continue;
    TreeMoves& u = p.up[(nodes[k].height - 1) / kTreeLevelsPerPass];
    u.tgt.push_back(k);
    for (int j : sources[k]) u.src.push_back((int)(255u << 24 | (unsigned)j));
    u.ptr.push_back((int)u.src.size());
  }

  p.formed.swap(used);
  std::fill(p.formed.begin(), p.formed.begin() + nc, 1);

  // downward: every cell from all its ancestors with a local expansion
  for (int c = 0; c < nc; c++) {
    p.down.tgt.push_back(c);
    for (int k = nodes[c].parent; k >= 0; k = nodes[k].parent)
      if (p.has_local[k]) p.down.src.push_back((int)(255u << 24 | (unsigned)k));
    p.down.ptr.push_back((int)p.down.src.size());
  }

  p.near.swap(near);
  make_near_lists(p, true, &p.sym);
  p.forward_slots = count_forward_slots(p);
  return true;
}

}  // namespace eb
