#include "mesh_host.h"

#include <algorithm>
#include <cmath>
#include <numeric>
#include <string>

#include "common.h"
#include "pairs.h"

namespace eb {

void target_split(int Q, int* K, int* nchunk)
{
  // Q <= 7 fits one item per triangle; larger rules are split into chunks of
  // at most 8 points (the last chunk padded with zero-weight points).
  if (Q <= 7) { *K = Q; *nchunk = 1; return; }
  *K = 8;
  *nchunk = (Q + 7) / 8;
}

int split_cells(int ncells)
{
  // larger ranges split at whole 128-triangle target tiles (4 cells); small
  // ones in the middle, so that no part is a sliver
  const int half = (ncells + 1) / 2;
  return ncells > 32 ? (half + 3) / 4 * 4 : half;
}

struct Centroid {
  double c[3];
  int i;
};

// Recursive bisection: t[0, n) is halved at a whole number of cells across
// the longest side of its box until one cell is left.
static void bisect(Centroid* t, int n)
{
  const int ncells = (n + kCell - 1) / kCell;
  if (ncells <= 1) return;
  double lo[3] = {t[0].c[0], t[0].c[1], t[0].c[2]}, hi[3] = {lo[0], lo[1], lo[2]};
  for (int k = 1; k < n; k++)
    for (int d = 0; d < 3; d++) {
      lo[d] = std::min(lo[d], t[k].c[d]);
      hi[d] = std::max(hi[d], t[k].c[d]);
    }
  int ax = 0;
  for (int d = 1; d < 3; d++)
    if (hi[d] - lo[d] > hi[ax] - lo[ax]) ax = d;
  const int m = split_cells(ncells) * kCell;  // < n: the right part holds at least one cell
  std::nth_element(t, t + m, t + n, [ax](const Centroid& a, const Centroid& b) {
    return a.c[ax] < b.c[ax] || (a.c[ax] == b.c[ax] && a.i < b.i);
  });
  bisect(t, m);
  bisect(t + m, n - m);
}

void vertex_ball(const HostMesh& m, int s0, int s1, double* ball)
{
  thread_local std::vector<d3> p;
  p.clear();
  for (int s = s0; s < s1; s++)
    for (int k = 0; k < 3; k++) {
      const double* v = &m.nodes[3 * (size_t)m.elems[3 * (size_t)m.perm[s] + k]];
      p.push_back(mk3(v[0], v[1], v[2]));
    }
  d3 lo = p[0], hi = p[0];
  for (const d3& v : p) {
    lo = mk3(std::min(lo.x, v.x), std::min(lo.y, v.y), std::min(lo.z, v.z));
    hi = mk3(std::max(hi.x, v.x), std::max(hi.y, v.y), std::max(hi.z, v.z));
  }
  d3 c = 0.5 * (lo + hi);
  double best = -1.0;
  for (int it = 0; it <= 4; it++) {
    double r2 = -1.0;
    d3 far = c;
    for (const d3& v : p) {
      const double e2 = dot3(v - c, v - c);
      if (e2 > r2) {
        r2 = e2;
        far = v;
      }
    }
    if (best < 0.0 || r2 < best) {
      best = r2;
      ball[0] = c.x;
      ball[1] = c.y;
      ball[2] = c.z;
    }
    c = c + (1.0 / (it + 4.0)) * (far - c);
  }
  ball[3] = std::sqrt(best) * (1.0 + 1e-12);
}

int prepare_host_mesh(int nv, const double* nodes, int ne, const int* elems1, int order, HostMesh* m,
                      bool topology)
{
  if (nv < 3 || ne < 1 || !nodes || !elems1)
    return set_error(EB_ERR_INVALID, "mesh needs >= 3 vertices, >= 1 triangle and non-null arrays");
  if (!make_quadrature(order, &m->quad))
    return set_error(EB_ERR_INVALID, "quadrature order must be in 0.." + std::to_string(kMaxOrder));
  m->nv = nv;
  m->ne = ne;
  m->order = order;
  m->Q = m->quad.nt;
  m->nodes.assign(nodes, nodes + 3 * (size_t)nv);
  m->elems.resize(3 * (size_t)ne);
  for (int i = 0; i < ne; i++) {
    for (int k = 0; k < 3; k++) {
      const int v = elems1[3 * i + k];
      if (v < 1 || v > nv)
        return set_error(EB_ERR_MESH, "triangle " + std::to_string(i) + " has vertex index " +
                                          std::to_string(v) + " outside 1.." + std::to_string(nv));
      m->elems[3 * i + k] = v - 1;
    }
    const int* f = &m->elems[3 * i];
    if (f[0] == f[1] || f[1] == f[2] || f[0] == f[2])
      return set_error(EB_ERR_MESH, "triangle " + std::to_string(i) + " repeats a vertex");
    const d3 a = mk3(nodes[3 * f[0]], nodes[3 * f[0] + 1], nodes[3 * f[0] + 2]);
    const d3 b = mk3(nodes[3 * f[1]], nodes[3 * f[1] + 1], nodes[3 * f[1] + 2]);
    const d3 c = mk3(nodes[3 * f[2]], nodes[3 * f[2] + 1], nodes[3 * f[2] + 2]);
    const d3 n = cross3(b - a, c - a);
    const double area2 = std::sqrt(dot3(n, n));
    const double scale = dot3(b - a, b - a) + dot3(c - a, c - a);
    if (!(area2 > 1e-14 * scale) || !std::isfinite(area2))
      return set_error(EB_ERR_MESH, "triangle " + std::to_string(i) + " is degenerate (zero area)");
  }

  // order by recursive bisection of the centroids
  std::vector<Centroid> cent(ne);
  for (int i = 0; i < ne; i++) {
    const int* f = &m->elems[3 * i];
    for (int d = 0; d < 3; d++) cent[i].c[d] = (nodes[3 * f[0] + d] + nodes[3 * f[1] + d] + nodes[3 * f[2] + d]) / 3.0;
    cent[i].i = i;
  }
  bisect(cent.data(), ne);
  m->perm.resize(ne);
  m->iperm.resize(ne);
  for (int s = 0; s < ne; s++) {
    m->perm[s] = cent[s].i;
    m->iperm[cent[s].i] = s;
  }
  m->ncells = (ne + kCell - 1) / kCell;
  m->cell_ball.resize(4 * (size_t)m->ncells);
  for (int c = 0; c < m->ncells; c++)
    vertex_ball(*m, c * kCell, std::min(ne, (c + 1) * kCell), &m->cell_ball[4 * (size_t)c]);
  target_split(m->Q, &m->K, &m->nchunk);
  m->nitems = ne * m->nchunk;
  if (topology) host_topology(m);
  return EB_OK;
}

void host_topology(HostMesh* m)
{
  const int nv = m->nv, ne = m->ne;
  // Vertex -> triangles.
  std::vector<int> vptr(nv + 1, 0), vtri(3 * (size_t)ne);
  for (int i = 0; i < 3 * ne; i++) vptr[m->elems[i] + 1]++;
  for (int v = 0; v < nv; v++) vptr[v + 1] += vptr[v];
  {
    std::vector<int> fill(vptr.begin(), vptr.end() - 1);
    for (int i = 0; i < ne; i++)
      for (int k = 0; k < 3; k++) vtri[fill[m->elems[3 * i + k]]++] = i;
  }

  // Near pairs per test triangle (sorted by trial index), DL slots per row.
  // Marks replace set operations: seen[j] = i once triangle j is a candidate of
  // row i, and slot[v] (with owner[v] = i) is vertex v's place in row i's
  // column list, so only the ~13 candidates and ~12 columns are sorted.
  const size_t guess = 14 * (size_t)ne;
  m->sl_rowptr.assign(ne + 1, 0);
  m->sl_col.clear();
  m->sl_col.reserve(guess);
  m->pair_i.clear();
  m->pair_i.reserve(guess);
  m->pair_kind.clear();
  m->pair_kind.reserve(guess);
  m->dl_rowptr.assign(ne + 1, 0);
  m->dl_col.clear();
  m->dl_col.reserve(guess);
  std::vector<int> seen(ne, -1), owner(nv, -1), slot(nv), cand, cols, first, entry_col;
  long long near_incl_repeat = 0;
  std::vector<int> contrib_ptr(1, 0), contrib;
  contrib_ptr.reserve(guess);
  contrib.reserve(3 * guess);
  for (int i = 0; i < ne; i++) {
    cand.clear();
    for (int k = 0; k < 3; k++) {
      const int v = m->elems[3 * i + k];
      for (int p = vptr[v]; p < vptr[v + 1]; p++)
        if (seen[vtri[p]] != i) {
          seen[vtri[p]] = i;
          cand.push_back(vtri[p]);
        }
    }
    std::sort(cand.begin(), cand.end());
    near_incl_repeat += (long long)cand.size();
    cols.clear();
    entry_col.clear();
    const int p0 = (int)m->sl_col.size();
    for (int j : cand) {
      const PairGeom g = classify_pair(&m->elems[3 * i], &m->elems[3 * j], i == j);
      if (g.kind == kPairRepeat) continue;  // a repeated triangle contributes nothing
      m->sl_col.push_back(j);
      m->pair_i.push_back(i);
      m->pair_kind.push_back((int8_t)g.kind);
      if (g.kind == kPairVertex || g.kind == kPairEdge) {
        int slots[3];
        dl_trial_slots(g, slots);
        for (int k = 0; k < 3; k++) {
          const int v = m->elems[3 * j + slots[k]];
          entry_col.push_back(v);
          if (owner[v] != i) {
            owner[v] = i;
            cols.push_back(v);
          }
        }
      } else {
        entry_col.insert(entry_col.end(), 3, -1);
      }
    }
    m->sl_rowptr[i + 1] = (int)m->sl_col.size();
    // entries 3 pair + k by column, ascending within each column
    std::sort(cols.begin(), cols.end());
    first.assign(cols.size() + 1, 0);
    for (size_t c = 0; c < cols.size(); c++) slot[cols[c]] = (int)c;
    for (int v : entry_col)
      if (v >= 0) first[slot[v] + 1]++;
    for (size_t c = 0; c < cols.size(); c++) {
      first[c + 1] += first[c];
      m->dl_col.push_back(cols[c]);
      contrib_ptr.push_back((int)contrib.size() + first[c + 1]);
    }
    const size_t base = contrib.size();
    contrib.resize(base + first[cols.size()]);
    for (size_t e = 0; e < entry_col.size(); e++)
      if (entry_col[e] >= 0) contrib[base + first[slot[entry_col[e]]]++] = 3 * p0 + (int)e;
    m->dl_rowptr[i + 1] = (int)m->dl_col.size();
  }
  m->dl_contrib_ptr.swap(contrib_ptr);
  m->dl_contrib.swap(contrib);
  m->far_quad_pairs = ((long long)ne * ne - near_incl_repeat) * (long long)m->Q * m->Q;
}

}  // namespace eb
