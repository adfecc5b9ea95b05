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

}  // namespace

bool make_tree_plan(const HostMesh& h, TreePlan* plan)
{
  TreePlan& p = *plan;
  const int nc = h.ncells;
  p.ncells = nc;
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
  p.ball.resize(nn);
  for (int c = 0; c < nc; c++) {
    const double* b = &h.cell_ball[4 * (size_t)c];
    p.ball[c] = dq{b[0], b[1], b[2], std::max(h.cell_rho[c], 1e-3 * b[3])};
  }
  // a move scales with the inverse distance of the two centres, so an inner
  // node's centre keeps away from those of its descendants (symmetric meshes
  // put them at the same point)
  std::function<bool(int, int)> clear = [&](int k, int j) {
    const dq &x = p.ball[k], &y = p.ball[j];
    const d3 v = mk3(x.x - y.x, x.y - y.y, x.z - y.z);
    const double s = kTreeMinStep * x.w;
    if (dot3(v, v) < s * s) return false;
    return nodes[j].left < 0 || (clear(k, nodes[j].left) && clear(k, nodes[j].right));
  };
  for (int k = nc; k < nn; k++) {
    const dq b = ball_of(p.ball, nodes[k].lo, nodes[k].hi);
    p.ball[k] = b;
    for (int t = 1; t < 64 && !(clear(k, nodes[k].left) && clear(k, nodes[k].right)); t++) {
      const double a = 2.4 * t, z = std::cos(1.7 * t), r = std::sqrt(1.0 - z * z), s = 0.004 * t * b.w;
      p.ball[k] = dq{b.x + s * r * std::cos(a), b.y + s * r * std::sin(a), b.z + s * z, b.w + s};
    }
  }

  // the tree against itself
  std::vector<std::pair<int, int>> far;
  std::vector<std::vector<int>> near(nc);  // later cells close to each cell
  const long long limit = std::max<long long>(4 * nc, (long long)nc * nc / 16);
  long long nnear = 0;
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
    const double s = (x.w + y.w) / kTreeTheta;
    if (dot3(d, d) > s * s) {
      far.push_back({a, b});
    } else if (A.left < 0 && B.left < 0) {
      near[std::min(a, b)].push_back(std::max(a, b));
      if (++nnear > limit) return false;
    } else if (B.left < 0 || (A.left >= 0 && x.w >= y.w)) {
      stack.push_back({A.left, b});
      stack.push_back({A.right, b});
    } else {
      stack.push_back({a, B.left});
      stack.push_back({a, B.right});
    }
  }

  // separated pairs in both directions, by target
  std::vector<int> count(nn + 1, 0);
  for (const auto& f : far) {
    count[f.first + 1]++;
    count[f.second + 1]++;
  }
  for (int k = 0; k < nn; k++) count[k + 1] += count[k];
  std::vector<int> fill(count.begin(), count.end() - 1), src(2 * far.size());
  std::vector<char> used(nn, 0);  // its multipole is read
  for (const auto& f : far) {
    src[fill[f.first]++] = f.second;
    src[fill[f.second]++] = f.first;
    used[f.first] = used[f.second] = 1;
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
  for (int k : order) {
    p.m2l.tgt.push_back(k);
    for (int q = count[k]; q < count[k + 1]; q++) {
      const dq &x = p.ball[k], &y = p.ball[src[q]];
      const d3 v = mk3(x.x - y.x, x.y - y.y, x.z - y.z);
      const double share = std::log(kTreeTheta) / std::log((x.w + y.w) / std::sqrt(dot3(v, v)));
      const int f = std::min(255, std::max(1, (int)std::ceil(255.0 * share)));
      p.m2l.src.push_back((int)((unsigned)f << 24 | (unsigned)src[q]));
    }
    std::sort(p.m2l.src.end() - (count[k + 1] - count[k]), p.m2l.src.end(),
              [](int a, int b) { return (unsigned)a >> 24 != (unsigned)b >> 24 ? (unsigned)a >> 24 > (unsigned)b >> 24 : a < b; });
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

  // downward: every cell from all its ancestors with a local expansion
  for (int c = 0; c < nc; c++) {
    p.down.tgt.push_back(c);
    for (int k = nodes[c].parent; k >= 0; k = nodes[k].parent)
      if (p.has_local[k]) p.down.src.push_back((int)(255u << 24 | (unsigned)k));
    p.down.ptr.push_back((int)p.down.src.size());
  }

  // close pairs: transposed slots first, then one forward slot per task, then
  // the far slot; the larger tasks first
  std::vector<std::vector<int>> all(nc);
  for (int c = 0; c < nc; c++) {
    std::sort(near[c].begin(), near[c].end());
    for (int j : near[c]) {
      all[c].push_back(j);
      all[j].push_back(c);
    }
  }
  auto lists = [&](const std::vector<std::vector<int>>& close, bool both, TreeNear& out) {
    std::vector<int> trans(nc, 0);
    if (both)
      for (int c = 0; c < nc; c++)
        for (int j : close[c]) trans[j]++;
    out.slot_off.assign(nc + 1, 0);
    for (int c = 0; c < nc; c++)
      out.slot_off[c + 1] =
          out.slot_off[c] + trans[c] + ((int)close[c].size() + kTreeNearChunk) / kTreeNearChunk + 1;
    std::vector<int> next(out.slot_off.begin(), out.slot_off.end() - 1);
    for (int c = 0; c < nc; c++) {
      const int e0 = (int)out.entries.size();
      out.entries.push_back(make_int2(c, -1));
      for (int j : close[c]) out.entries.push_back(make_int2(j, both ? next[j]++ : -1));
      const int e1 = (int)out.entries.size();
      int slot = out.slot_off[c] + trans[c];
      for (int e = e0; e < e1; e += kTreeNearChunk)
        out.tasks.push_back(make_int4(c, e, std::min(e1, e + kTreeNearChunk), slot++));
    }
    std::stable_sort(out.tasks.begin(), out.tasks.end(),
                     [](const int4& a, const int4& b) { return a.z - a.y > b.z - b.y; });
  };
  lists(near, true, p.sym);
  lists(all, false, p.fwd);
  return true;
}

}  // namespace eb
