// Tree far field: the sum over all pairs of quadrature points in time
// proportional to their number (rules of 7 points, and of 8 and more).
//
// Clusters of triangles (the nodes of the bisection that orders the mesh) are
// paired as in tree_plan.h. Between separated clusters the kernel 1/|x - y| is
// expanded in solid harmonics; close cells are summed point by point with the
// inner loops of the symmetric far field. Harmonics are normalised so that
// rotations act unitarily (C = sqrt(4 pi / (2n + 1)) Y):
//
//   R_n^m(x) = |x|^n C_n^m,   S_n^m(x) = |x|^-(n+1) C_n^m,
//   1/|x - y| = sum_nm conj(R_n^m(y)) S_n^m(x),  |y| < |x|,
//
// a cluster's multipole is A_n^m = sum q R_n^m(y - c) / rho^n (rho its radius;
// every stored coefficient is of the size of the charges whatever the mesh's
// units), a double-layer source of strength s and normal n enters as
// s (n.grad) R_n^m, and a local expansion gives phi = Re sum L_n^m conj(R_n^m).
// Only m >= 0 is kept (the sums are real).
//
//   points -> multipoles   tree_p2m_kernel   one CTA per cell
//   multipoles upward      tree_move_kernel<kUp>, three levels per launch
//   multipoles -> locals   tree_move_kernel<kAcross>
//   locals downward        tree_move_kernel<kDown>, all ancestors at once
//   locals -> points       tree_l2p_kernel, into the last partial slot
//   close cells            tree_near_kernel, one warp per task
//
// Moving an expansion along a vector d costs 2 p^3 multiply-adds instead of
// p^4: it is rotated so that d becomes the z axis, moved along z (which
// couples only equal m) and rotated back. The rotation about y splits into
// rotations about z (a phase per m) and the constant rotation about y by 90
// degrees: Ry(90) Rz(theta) Ry(-90) Rz(90 - phi) takes d to z. The matrix of
// Ry(90) couples only half of the orders of a degree, real and imaginary
// parts apart, and that of Ry(-90) differs by a sign per degree.
//
// Every sum runs in a fixed order on fixed lanes and every slot has one
// writer, so results are bitwise reproducible.
#include "farfield_tree.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <numeric>
#include <type_traits>

#include "farfield_sym_eval.cuh"

namespace eb {

namespace {

enum Move { kUp, kAcross, kDown };

// Constant tables of one order (device pointers). The matrices are stored as
// mma operand fragments: lane l holds output slot 8 t + (l / 8) + 4 (l / 4 % 2)
// and input slot 4 k + l % 4 of tile t and step k (zeros outside):
//   Ry(90), per degree: [part][output parity][t][k], slots as in the kernel;
//   along z, per order m: [t][k], slot = n - m.
struct TreeTables {
  const double *bmat, *tmat[3];
  const int* pair;     // (n, m): m | n << 8
  const double2* rec;  // (n, m): R_n^m = rec.x z R_{n-1}^m - rec.y r^2 R_{n-2}^m (n > m);
                       // (m, m): R_m^m = rec.x (x + i y) R_{m-1}^{m-1}
};

__device__ __forceinline__ int tree_pair(int n, int m) { return n * (n + 1) / 2 + m; }

// Block b's entry among the meshes and its index there.
__device__ __forceinline__ int tree_entry(const int* __restrict__ off, int n, int& b)
{
  if (n == 1) return 0;
  int lo = 0, hi = n;  // off[lo] <= b < off[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (off[mid] <= b) lo = mid;
    else hi = mid;
  }
  b -= off[lo];
  return lo;
}

// ---------------------------------------------------------------------------
// Moves. A CTA owns one target node and takes its sources eight at a time; an
// mma m8n8k4 multiplies the eight sources' coefficients (rows) with eight
// outputs of a constant matrix, for every column. A warp owns whole degrees
// for the rotations and whole orders for the move along z:
//
//   per degree  load, phase, Ry(-90), phase, Ry(90)     -> shared memory
//   per order   along z, in place
//   per degree  Ry(-90), phase, Ry(90), phase           -> running sums
//
// A pair whose radii are small against its distance needs fewer degrees: those
// beyond its order (TreeMoves::src) are left out of all stages.
//
// The result fragment of an mma (a lane has source lane / 4, outputs 2j and
// 2j + 1, j = lane % 4) is the operand fragment of the next one when the
// output columns stand for slots j and j + 4, so the chain of a degree stays
// in registers. Coefficient slots of one parity of m: m = 2 slot + parity,
// slot = 4 el + j; real and imaginary parts sit in the same slots (the
// imaginary part of m = 0 is a zero row and column).
//
// Measured on the SL+DL apply at 81,920 triangles (105,000 moves, two columns;
// mixed / FP64): one warp per source with scalar multiply-adds 3.5 / 39 ms
// (order 30); batched vectors, a lane per output 3.0 / 12.3 (the shared-memory
// pipe 95 % busy: two wavefronts per 32 products); mma with all stages through
// shared memory 3.4 / 13.0 (latency of the matrix loads); chains in registers
// 2.55 / 12.1; degrees by separation 2.50 / 10.8; degrees specialised by parity
// and size, so that slots are not selected at run time, 2.17 / 8.8. The mma
// pipe itself sustains 64 multiply-adds per clock and SM, as DFMA does.

constexpr int kBatch = 8;  // sources of a batch

template <int P, int NC>
struct MoveShape {
  // Larger orders: two columns share the matrix loads of one CTA of eight
  // warps (113 KB); a single column runs two CTAs of four. Measured, 81,920
  // triangles, SL+DL FP64: 8.78 ms against 8.96 with a column per CTA.
  static constexpr int kWarps = P > 16 && NC == 2 ? 8 : 4;
  static constexpr int kCtas = P <= 16 ? 3 : NC == 2 ? 1 : 2;
  static constexpr int kThreads = 32 * kWarps;
  static constexpr int kEls = 2 * ((P / 2 + 8) / 8);  // slot groups of four per parity, even
  static constexpr int kRows = 2 * tree_pairs(P);     // real rows m-major, then imaginary rows
  static constexpr size_t smem() { return sizeof(double) * (kBatch + 1) * kRows * NC; }
};

__device__ __forceinline__ void mma_f64(double& c0, double& c1, double a, double b)
{
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c0), "+d"(c1)
      : "d"(a), "d"(b));
}

__host__ __device__ constexpr int order_row(int P, int m) { return m * (P + 1) - m * (m - 1) / 2; }  // of (m, m)

// Slots of a parity in degree n.
__device__ __forceinline__ int slots_of(int n, int par) { return par ? (n + 1) >> 1 : (n >> 1) + 1; }

// b^k by squaring, k < 32
__device__ __forceinline__ double power(double b, int k)
{
  double r = 1.0;
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    if (k >> i & 1) r *= b;
    b *= b;
  }
  return r;
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__device__ __forceinline__ double2 power(double2 b, int k)
{
  double2 r = make_double2(1.0, 0.0);
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    if (k >> i & 1) r = cmul(r, b);
    b = cmul(b, b);
  }
  return r;
}

// e[par][el] = base^m of this lane's slots.
template <int E>
__device__ __forceinline__ void lane_phases(double2 base, int j, double2 (&e)[2][E])
{
  const double2 b2 = cmul(base, base), b4 = cmul(b2, b2), b8 = cmul(b4, b4);
  e[0][0] = power(b2, j);
#pragma unroll
  for (int el = 0; el < E; ++el) {
    if (el > 0) e[0][el] = cmul(e[0][el - 1], b8);
    e[1][el] = cmul(e[0][el], base);
  }
}

// One degree's coefficients of NC columns: real and imaginary parts, parity, slot group.
template <int NC, int E>
struct Degree {
  double x[NC][2][2][E];
};

// x = Ry(90) x for a degree n of parity ODD with at most 4 EN slots per parity
// (frag: its matrix, stored for E slot groups).
template <int NC, int E, int EN, int ODD>
__device__ __forceinline__ void turn(const double* __restrict__ frag, int n, Degree<NC, EN>& d)
{
  Degree<NC, EN> y;
#pragma unroll
  for (int part = 0; part < 2; ++part)
#pragma unroll
    for (int par = 0; par < 2; ++par) {
      constexpr int kTiles = (EN + 1) / 2;
      const int from = (ODD + par + part) & 1;
      const bool last = slots_of(n, from) > 4 * (EN - 1);  // the last step has inputs
#pragma unroll
      for (int t = 0; t < kTiles; ++t) {
        double c0[NC], c1[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) c0[c] = c1[c] = 0.0;
        const double* f = frag + (((part * 2 + par) * (E / 2) + t) * E) * 32;
#pragma unroll
        for (int k = 0; k < EN; ++k)
          if (k < EN - 1 || EN == 1 || last) {
            const double b = __ldg(f + 32 * k);
#pragma unroll
            for (int c = 0; c < NC; ++c) mma_f64(c0[c], c1[c], d.x[c][part][from][k], b);
          }
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          y.x[c][part][par][2 * t] = c0[c];
          if (2 * t + 1 < EN) y.x[c][part][par][2 * t + 1] = c1[c];
        }
      }
    }
  d = y;
}

// x = scale x e^{+-i m alpha}; MIRROR: of (re, -im) (Ry(-90) is Ry(90) times
// (-1)^n for real and -(-1)^n for imaginary parts)
template <int NC, int E, int EN, int SIGN, bool MIRROR>
__device__ __forceinline__ void phase(const double2 (&e)[2][E], double scale, Degree<NC, EN>& d)
{
#pragma unroll
  for (int par = 0; par < 2; ++par)
#pragma unroll
    for (int el = 0; el < EN; ++el) {
      const double fr = MIRROR ? e[par][el].x : scale * e[par][el].x, fi = MIRROR ? e[par][el].y : scale * e[par][el].y;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const double re = d.x[c][0][par][el], im = d.x[c][1][par][el];
        const double si = (MIRROR ? -1.0 : 1.0) * SIGN, sc = MIRROR ? -1.0 : 1.0, ss = SIGN;
        d.x[c][0][par][el] = re * fr - si * (im * fi);
        d.x[c][1][par][el] = ss * (re * fi) + sc * (im * fr);
      }
    }
}

// Stage of a degree before the move along z: coefficients a (pair (n, 0) of
// column 0) into the rows of zb.
template <int P, int NC, int EN, int ODD>
__device__ __forceinline__ void before_z(const TreeTables& tab, int n, bool on, const double2* __restrict__ a,
                                         size_t cstride, const double2 (&ephi)[2][MoveShape<P, NC>::kEls],
                                         const double2 (&eth)[2][MoveShape<P, NC>::kEls], double scale, int vec, int j,
                                         int lane, double* zb)
{
  using Mv = MoveShape<P, NC>;
  constexpr int E = Mv::kEls, kPairs = tree_pairs(P);
  Degree<NC, EN> x;
#pragma unroll
  for (int par = 0; par < 2; ++par)
#pragma unroll
    for (int el = 0; el < EN; ++el) {
      const int m = 2 * (4 * el + j) + par;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const double2 v = on && m <= n ? a[c * cstride + m] : make_double2(0.0, 0.0);
        x.x[c][0][par][el] = v.x;
        x.x[c][1][par][el] = v.y;
      }
    }
  const double* frag = tab.bmat + (size_t)n * (2 * E * E) * 32 + lane;
  phase<NC, E, EN, 1, false>(ephi, ODD ? -scale : scale, x);
  turn<NC, E, EN, ODD>(frag, n, x);
  phase<NC, E, EN, 1, true>(eth, 1.0, x);
  turn<NC, E, EN, ODD>(frag, n, x);
#pragma unroll
  for (int par = 0; par < 2; ++par)
#pragma unroll
    for (int el = 0; el < EN; ++el) {
      const int m = 2 * (4 * el + j) + par;
      if (m <= n) {
        double* r = zb + (order_row(P, m) + n - m) * kBatch + vec;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          r[c * Mv::kRows * kBatch] = x.x[c][0][par][el];
          r[(c * Mv::kRows + kPairs) * kBatch] = x.x[c][1][par][el];
        }
      }
    }
}

// Stage of a degree after the move along z: rows of zb turned back, added over
// the eight sources and onto acc ([column][part][pair]).
template <int P, int NC, int EN, int ODD>
__device__ __forceinline__ void after_z(const TreeTables& tab, int n, const double2 (&ephi)[2][MoveShape<P, NC>::kEls],
                                        const double2 (&eth)[2][MoveShape<P, NC>::kEls], double scale, int vec, int j,
                                        int lane, const double* zb, double* acc)
{
  using Mv = MoveShape<P, NC>;
  constexpr int E = Mv::kEls, kPairs = tree_pairs(P);
  Degree<NC, EN> x;
#pragma unroll
  for (int par = 0; par < 2; ++par)
#pragma unroll
    for (int el = 0; el < EN; ++el) {
      const int m = 2 * (4 * el + j) + par;
      const double* r = zb + (order_row(P, m) + n - m) * kBatch + vec;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        x.x[c][0][par][el] = m <= n ? r[c * Mv::kRows * kBatch] : 0.0;
        x.x[c][1][par][el] = m <= n ? r[(c * Mv::kRows + kPairs) * kBatch] : 0.0;
      }
    }
  const double* frag = tab.bmat + (size_t)n * (2 * E * E) * 32 + lane;
  turn<NC, E, EN, ODD>(frag, n, x);
  phase<NC, E, EN, -1, true>(eth, 1.0, x);
  turn<NC, E, EN, ODD>(frag, n, x);
  phase<NC, E, EN, -1, false>(ephi, ODD ? -scale : scale, x);
  // halving the values per lane at each step: lane bit 4 keeps the part, bit 3
  // the parity, bit 2 the slot group's low bit
  const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    double u[2][EN], w[EN];
#pragma unroll
    for (int par = 0; par < 2; ++par)
#pragma unroll
      for (int el = 0; el < EN; ++el) {
        const double keep = b4 ? x.x[c][1][par][el] : x.x[c][0][par][el];
        const double give = b4 ? x.x[c][0][par][el] : x.x[c][1][par][el];
        u[par][el] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
      }
#pragma unroll
    for (int el = 0; el < EN; ++el) {
      const double keep = b3 ? u[1][el] : u[0][el], give = b3 ? u[0][el] : u[1][el];
      w[el] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
    }
    double* to = acc + (2 * c + (lane >> 4)) * kPairs + tree_pair(n, 0);
    if constexpr (EN == 1) {
      const double v = w[0] + __shfl_xor_sync(0xffffffffu, w[0], 4);
      const int m = 2 * j + (lane >> 3 & 1);
      if (!b2 && m <= n) to[m] += v;
    } else {
#pragma unroll
      for (int i = 0; i < EN / 2; ++i) {
        const double keep = b2 ? w[2 * i + 1] : w[2 * i], give = b2 ? w[2 * i] : w[2 * i + 1];
        const double v = keep + __shfl_xor_sync(0xffffffffu, give, 4);
        const int m = 2 * (4 * (2 * i + (lane >> 2 & 1)) + j) + (lane >> 3 & 1);
        if (m <= n) to[m] += v;
      }
    }
  }
}

template <int P, int NC, int MODE>
__global__ void __launch_bounds__(MoveShape<P, NC>::kThreads, MoveShape<P, NC>::kCtas)
    tree_move_kernel(const TreeDesc* __restrict__ descs, const int* __restrict__ off, int nmesh, int pass, TreeTables tab)
{
  using Mv = MoveShape<P, NC>;
  constexpr int kPairs = tree_pairs(P), W = Mv::kWarps, E = Mv::kEls, KT = (P + 4) / 4;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* zb = reinterpret_cast<double*>(smem_raw);     // [column][row][source]
  double* acc = zb + (size_t)kBatch * Mv::kRows * NC;   // [column][part][pair]
  int node = blockIdx.x;
  const TreeDesc& d = descs[tree_entry(off, nmesh, node)];
  if (d.far.active && *d.far.active == 0) return;
  const TreeMovesDev mv = MODE == kUp ? d.up[pass] : MODE == kAcross ? d.m2l : d.down;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, vec = lane >> 2, j = lane & 3;
  for (int i = threadIdx.x; i < 2 * NC * kPairs; i += Mv::kThreads) acc[i] = 0.0;
  const int tgt = mv.tgt[node];
  const dq bt = d.ball[tgt];
  const size_t cstride = (size_t)d.nnodes * kPairs, col0 = blockIdx.y * NC * cstride;
  const double2* from = (MODE == kDown ? d.local : d.multipole) + col0;
  const int n0 = (P - warp) % W;  // this warp's degrees: n0, n0 + W, ...
  __syncthreads();

  const int end = mv.ptr[node + 1];
#pragma unroll 1
  for (int first = mv.ptr[node]; first < end; first += kBatch) {
    const bool on = first + vec < end;
    const int entry = mv.src[on ? first + vec : first];
    // the batch runs to the highest order that one of its pairs needs
    const int order = ((P + 1) * (int)__reduce_max_sync(0xffffffffu, (unsigned)entry >> 24) + 254) / 255 - 1;
    const int src = entry & 0xffffff;
    const dq bs = d.ball[src];
    const double2* a = from + (size_t)src * kPairs;
    // the vector that becomes the z axis: from the source's centre to the
    // target's, reversed for a multipole (its points move the other way)
    const double sg = MODE == kUp ? -1.0 : 1.0;
    const double dx = sg * (bt.x - bs.x), dy = sg * (bt.y - bs.y), dz = sg * (bt.z - bs.z);
    const double h2 = dx * dx + dy * dy, h = sqrt(h2), dist = sqrt(h2 + dz * dz);
    const double rd = 1.0 / dist, rh = h > 0.0 ? 1.0 / h : 0.0;
    double2 ephi[2][E], eth[2][E];
    lane_phases(h > 0.0 ? make_double2(dy * rh, dx * rh) : make_double2(0.0, 1.0), j, ephi);  // e^{i (90 - phi)}
    lane_phases(make_double2(dz * rd, h * rd), j, eth);
    // degrees scale with the radii their coefficients are stored for and with
    // the step: to the power -n on the side of irregular or moved multipoles,
    // n on the other
    const double in = MODE == kDown ? dist / bs.w : bs.w * rd;
    const double out = MODE == kUp ? dist / bt.w : bt.w * rd;
    double scale = power(in, n0), step = power(in, W);
#pragma unroll 1
    for (int n = n0; n <= order; n += W, scale *= step) {
      const double2* an = a + tree_pair(n, 0);
      if (n < 4 * E) {  // half of the slot groups
        if (n & 1) before_z<P, NC, E / 2, 1>(tab, n, on, an, cstride, ephi, eth, scale, vec, j, lane, zb);
        else before_z<P, NC, E / 2, 0>(tab, n, on, an, cstride, ephi, eth, scale, vec, j, lane, zb);
      } else {
        if (n & 1) before_z<P, NC, E, 1>(tab, n, on, an, cstride, ephi, eth, scale, vec, j, lane, zb);
        else before_z<P, NC, E, 0>(tab, n, on, an, cstride, ephi, eth, scale, vec, j, lane, zb);
      }
    }
    __syncthreads();

#pragma unroll 1
    for (int q = 0; q * W <= order; ++q) {
      const int m = q & 1 ? (q + 1) * W - 1 - warp : q * W + warp;
      if (m > order) continue;
      const int len = order + 1 - m, steps = (len + 3) >> 2, tiles = (len + 7) >> 3;
      const double* frag = tab.tmat[MODE] + (size_t)m * (KT * ((KT + 1) / 2)) * 32 + lane;
      double* r = zb + (order_row(P, m) + j) * kBatch + vec;
      double a2[NC][2][KT];
#pragma unroll
      for (int k = 0; k < KT; ++k)
        if (k < steps) {
          const bool in_range = 4 * k + j < len;
#pragma unroll
          for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int part = 0; part < 2; ++part)
              a2[c][part][k] = in_range ? r[(c * Mv::kRows + part * kPairs + 4 * k) * kBatch] : 0.0;
        }
#pragma unroll
      for (int t = 0; t < (KT + 1) / 2; ++t)
        if (t < tiles) {
          double y[NC][2][2];
#pragma unroll
          for (int c = 0; c < NC; ++c) y[c][0][0] = y[c][0][1] = y[c][1][0] = y[c][1][1] = 0.0;
#pragma unroll
          for (int k = 0; k < KT; ++k)
            if (k < steps) {
              const double b = __ldg(frag + (t * KT + k) * 32);
#pragma unroll
              for (int c = 0; c < NC; ++c) {
                mma_f64(y[c][0][0], y[c][0][1], a2[c][0][k], b);
                mma_f64(y[c][1][0], y[c][1][1], a2[c][1][k], b);
              }
            }
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (8 * t + 4 * h + j < len)
#pragma unroll
              for (int c = 0; c < NC; ++c) {
                r[(c * Mv::kRows + 8 * t + 4 * h) * kBatch] = y[c][0][h];
                r[(c * Mv::kRows + kPairs + 8 * t + 4 * h) * kBatch] = y[c][1][h];
              }
        }
    }
    __syncthreads();

    scale = on ? (MODE == kAcross ? rd : 1.0) * power(out, n0) : 0.0;
    step = power(out, W);
#pragma unroll 1
    for (int n = n0; n <= order; n += W, scale *= step) {
      if (n < 4 * E) {
        if (n & 1) after_z<P, NC, E / 2, 1>(tab, n, ephi, eth, scale, vec, j, lane, zb, acc);
        else after_z<P, NC, E / 2, 0>(tab, n, ephi, eth, scale, vec, j, lane, zb, acc);
      } else {
        if (n & 1) after_z<P, NC, E, 1>(tab, n, ephi, eth, scale, vec, j, lane, zb, acc);
        else after_z<P, NC, E, 0>(tab, n, ephi, eth, scale, vec, j, lane, zb, acc);
      }
    }
    __syncthreads();
  }
  const bool add = MODE == kDown && d.has_local[tgt];
  double2* to = (MODE == kUp ? d.multipole : d.local) + col0 + (size_t)tgt * kPairs;
  for (int it = threadIdx.x; it < NC * kPairs; it += Mv::kThreads) {
    const int c = it / kPairs, i = it - c * kPairs;
    double2* t = to + c * cstride + i;
    const double2 old = add ? *t : make_double2(0.0, 0.0);
    *t = make_double2(old.x + acc[2 * c * kPairs + i], old.y + acc[(2 * c + 1) * kPairs + i]);
  }
}

// ---------------------------------------------------------------------------
// Points and expansions. Four warps per cell, one lane per triangle with its
// seven points in registers; a warp runs every fourth order m of the
// recurrences in n, back and forth (orders 0, 7, 8, ... for warp 0) so that all
// warps have the same number of degrees. Both directions use w_a-weighted sums
// over a triangle's points: sources need sum_b q_b R(y_b), targets sum_a w_a
// phi(x_a). Latency of the recurrence and of the lane sums bounds them. SL+DL
// apply at 81,920 triangles, mixed / FP64: orders in turn and the factors of
// R_m^m computed 2.162 / 8.74 ms, even shares and tabulated factors 2.125 /
// 8.68; eight warps per cell 2.27 / 8.92.

constexpr int kCellWarps = 4;
constexpr int kSumRows = 8, kSumStride = 36;  // conflict-free rows of the lane sums

constexpr int kWideItem = 8;  // target points per item of rules of more than 7
constexpr int kWideTile = 8;  // source triangles staged at a time for those rules (even)

struct CellPoints {
  double x[kQ], y[kQ], z[kQ], r2[kQ];
};

// Points first .. first + kQ of a rule of Q (the last repeated past its end).
__device__ __forceinline__ void load_points(const TreeDesc& d, int tri, double inv_rho, CellPoints& p, int Q = kQ,
                                            int first = 0)
{
#pragma unroll
  for (int a = 0; a < kQ; ++a) {
    const dq q = d.pos[(size_t)tri * Q + min(first + a, Q - 1)];
    p.x[a] = -0.5 * q.x * inv_rho;
    p.y[a] = -0.5 * q.y * inv_rho;
    p.z[a] = -0.5 * q.z * inv_rho;
    p.r2[a] = p.x[a] * p.x[a] + p.y[a] * p.y[a] + p.z[a] * p.z[a];
  }
}

// Runs fn(n, m, re, im) over degrees n = m .. P of this warp's orders m, with
// the harmonics of the kQ points in re, im.
template <int P, typename F>
__device__ __forceinline__ void each_harmonic(const TreeTables& tab, const CellPoints& p, int warp, F&& fn)
{
  double dr[kQ], di[kQ];  // R_m^m
#pragma unroll
  for (int a = 0; a < kQ; ++a) {
    dr[a] = 1.0;
    di[a] = 0.0;
  }
#pragma unroll 1
  for (int m = 0; m <= P; ++m) {
    if (m > 0) {
      const double f = tab.rec[tree_pair(m, m)].x;
#pragma unroll
      for (int a = 0; a < kQ; ++a) {
        const double t = f * (p.x[a] * dr[a] - p.y[a] * di[a]);
        di[a] = f * (p.x[a] * di[a] + p.y[a] * dr[a]);
        dr[a] = t;
      }
    }
    const int w = m & (kCellWarps - 1);
    if ((m & kCellWarps ? kCellWarps - 1 - w : w) != warp) continue;
    double r1[kQ], i1[kQ], r0[kQ], i0[kQ];
#pragma unroll
    for (int a = 0; a < kQ; ++a) {
      r1[a] = dr[a];
      i1[a] = di[a];
      r0[a] = i0[a] = 0.0;
    }
    fn(m, m, r1, i1);
#pragma unroll 1
    for (int n = m + 1; n <= P; ++n) {
      const double2 c = tab.rec[tree_pair(n, m)];
#pragma unroll
      for (int a = 0; a < kQ; ++a) {
        const double az = c.x * p.z[a], br = c.y * p.r2[a];
        const double tr = az * r1[a] - br * r0[a], ti = az * i1[a] - br * i0[a];
        r0[a] = r1[a];
        i0[a] = i1[a];
        r1[a] = tr;
        i1[a] = ti;
      }
      fn(n, m, r1, i1);
    }
  }
}

// Multipoles of one cell: NSL single-layer columns (they share sum_b w_b J
// R(y_b)), and for ND = 1 the double-layer column blockIdx.y. KIND: both apart,
// single minus double layer in one column (the representation formula), or
// the strengths of the double-layer column as charges (P1 single layer).
// WIDE: a rule of more than kQ points, kQ at a time.
enum Sources { kApart, kDiff, kCharges };
template <int P, int NSL, int ND, int KIND = kApart, bool WIDE = false>
__global__ void __launch_bounds__(32 * kCellWarps)
    tree_p2m_kernel(const TreeDesc* __restrict__ descs, const int* __restrict__ off, int nmesh, ApplyArgs one,
                    const ApplyArgs* __restrict__ many, TreeTables tab)
{
  constexpr int kPairs = tree_pairs(P);
  constexpr int kRows = KIND == kCharges ? 2 : 2 * NSL + 6 * ND;
  static_assert(kRows <= kSumRows, "one row of lane sums per value");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* s_red = reinterpret_cast<double*>(smem_raw) + (threadIdx.x >> 5) * kSumRows * kSumStride;
  double* s_sum = reinterpret_cast<double*>(smem_raw) + kCellWarps * kSumRows * kSumStride;  // [kRows][kPairs]
  int cell = blockIdx.x;
  const int e = tree_entry(off, nmesh, cell);
  const TreeDesc& d = descs[e];
  if (d.far.active && *d.far.active == 0) return;
  const ApplyArgs& A = many ? many[e] : one;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double rho = d.ball[cell].w;
  const int tri = cell * kCell + lane;
  const bool on = tri < A.ne;
  const int sel = on ? tri : cell * kCell;
  double t[NSL > 0 ? NSL : 1], nrm[3] = {0.0, 0.0, 0.0}, u0 = 0.0, u1 = 0.0, u2 = 0.0;
  const int orig = A.perm[sel];
#pragma unroll
  for (int c = 0; c < NSL; ++c) t[c] = A.t[(size_t)c * A.tstride + orig];
  if constexpr (ND > 0) {
    const int4 v = A.svid[sel];
    const double* u = A.u + (size_t)blockIdx.y * A.ustride;
    u0 = u[v.x]; u1 = u[v.y]; u2 = u[v.z];
    const dq n = A.trin[sel];
    nrm[0] = n.x; nrm[1] = n.y; nrm[2] = n.z;
  }
  const int Q = WIDE ? A.Q : kQ;
#pragma unroll 1
  for (int first = 0; first < Q; first += kQ) {
    CellPoints p;
    load_points(d, sel, 1.0 / rho, p, Q, first);
    double wj[kQ], s[kQ];
#pragma unroll
    for (int a = 0; a < kQ; ++a) {
      const int b = min(first + a, Q - 1);
      wj[a] = on && first + a < Q ? A.wj[(size_t)sel * Q + b] : 0.0;
      const double e1 = A.bary[2 * b], e2 = A.bary[2 * b + 1];
      s[a] = wj[a] * ((1.0 - e1 - e2) * u0 + e1 * u1 + e2 * u2);
    }
    each_harmonic<P>(tab, p, warp, [&](int n, int m, const double (&re)[kQ], const double (&im)[kQ]) {
      int row = 0;
      if constexpr (NSL > 0) {
        double hr = 0.0, hi = 0.0;
#pragma unroll
        for (int a = 0; a < kQ; ++a) {
          hr += wj[a] * re[a];
          hi += wj[a] * im[a];
        }
#pragma unroll
        for (int c = 0; c < NSL; ++c) {
          s_red[row++ * kSumStride + lane] = hr * t[c];
          s_red[row++ * kSumStride + lane] = hi * t[c];
        }
      }
      if constexpr (ND > 0) {
        double gr = 0.0, gi = 0.0;
#pragma unroll
        for (int a = 0; a < kQ; ++a) {
          gr += s[a] * re[a];
          gi += s[a] * im[a];
        }
        if constexpr (KIND == kCharges) {
          s_red[lane] = gr;
          s_red[kSumStride + lane] = gi;
        } else {
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            s_red[row++ * kSumStride + lane] = gr * nrm[k];
            s_red[row++ * kSumStride + lane] = gi * nrm[k];
          }
        }
      }
      __syncwarp();
      // four lanes add a row of 32
      const int r = lane >> 2, part = lane & 3;
      double v = 0.0;
      if (r < kRows)
#pragma unroll
        for (int k = 0; k < 8; ++k) v += s_red[r * kSumStride + part + 4 * k];
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      if (part == 0 && r < kRows) {
        double* sum = &s_sum[r * kPairs + tree_pair(n, m)];
        *sum = WIDE && first ? *sum + v : v;  // the same thread every time
      }
      __syncwarp();
    });
  }
  __syncthreads();
  const size_t cstride = (size_t)d.nnodes * kPairs;
  double2* out = d.multipole + (size_t)cell * kPairs;
  for (int i = threadIdx.x; i < kPairs; i += 32 * kCellWarps) {
    if constexpr (KIND == kApart)
#pragma unroll
      for (int c = 0; c < NSL; ++c)
        out[c * cstride + i] = make_double2(s_sum[2 * c * kPairs + i], s_sum[(2 * c + 1) * kPairs + i]);
    if constexpr (KIND == kCharges) {
      out[i] = make_double2(s_sum[i], s_sum[kPairs + i]);
    } else if constexpr (ND > 0) {
      // (n.grad) R_n^m from the moments G^k = sum s n_k R of degree n - 1
      const double* g = s_sum + 2 * NSL * kPairs;
      const int info = tab.pair[i];
      const int m = info & 255, n = info >> 8;
      double ar = 0.0, ai = 0.0;
      if (n > 0) {
        if (m < n) {
          const int j = tree_pair(n - 1, m);
          const double f = sqrt((double)((n - m) * (n + m)));
          ar += f * g[4 * kPairs + j];
          ai += f * g[5 * kPairs + j];
        }
        {  // -1/2 (G^x + i G^y)_{n-1}^{m-1}
          const double f = -0.5 * sqrt((double)((n + m) * (n + m - 1)));
          double xr = 0.0, xi = 0.0, yr = 0.0, yi = 0.0;
          if (m > 0) {
            const int j = tree_pair(n - 1, m - 1);
            xr = g[j]; xi = g[kPairs + j]; yr = g[2 * kPairs + j]; yi = g[3 * kPairs + j];
          } else if (n > 1) {  // order -1: minus the conjugate of order 1
            const int j = tree_pair(n - 1, 1);
            xr = -g[j]; xi = g[kPairs + j]; yr = -g[2 * kPairs + j]; yi = g[3 * kPairs + j];
          }
          ar += f * (xr - yi);
          ai += f * (xi + yr);
        }
        if (m + 1 < n) {  // +1/2 (G^x - i G^y)_{n-1}^{m+1}
          const double f = 0.5 * sqrt((double)((n - m) * (n - m - 1)));
          const int j = tree_pair(n - 1, m + 1);
          ar += f * (g[j] + g[3 * kPairs + j]);
          ai += f * (g[kPairs + j] - g[2 * kPairs + j]);
        }
        ar /= rho;
        ai /= rho;
      }
      if constexpr (KIND == kDiff) out[i] = make_double2(s_sum[i] - ar, s_sum[kPairs + i] - ai);
      else out[((size_t)NSL + blockIdx.y) * cstride + i] = make_double2(ar, ai);
    }
  }
}

template <int P, int NSL, int ND>
constexpr size_t p2m_smem()
{
  return sizeof(double) * (kCellWarps * kSumRows * kSumStride + (2 * NSL + 6 * ND) * tree_pairs(P));
}

// Far sums of one cell's rows: sum_a w_a phi_c(x_a) for every column c; P1T:
// sum_a w_a phi_k(x_a) phi(x_a) of one column with the triangle's three hat
// functions. WIDE: a rule of more than kQ points, kQ at a time.
template <int P, int NC, bool P1T = false, bool WIDE = false>
__global__ void __launch_bounds__(32 * kCellWarps)
    tree_l2p_kernel(const TreeDesc* __restrict__ descs, const int* __restrict__ off, int nmesh, TreeTables tab)
{
  constexpr int kPairs = tree_pairs(P);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* s_loc = reinterpret_cast<double2*>(smem_raw);  // [NC][kPairs]
  constexpr int NO = P1T ? 3 : NC;
  __shared__ double s_part[kCellWarps][NO][kCell];
  int cell = blockIdx.x;
  const TreeDesc& d = descs[tree_entry(off, nmesh, cell)];
  if (d.far.active && *d.far.active == 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < kPairs * NC; i += 32 * kCellWarps) {
    const int c = i / kPairs, q = i - c * kPairs;
    double2 v = d.local[((size_t)c * d.nnodes + cell) * kPairs + q];
    if (tab.pair[q] & 255) {  // orders m and -m
      v.x *= 2.0;
      v.y *= 2.0;
    }
    s_loc[i] = v;
  }
  const int tri = cell * kCell + lane;
  const bool on = tri < d.far.ne;
  const int sel = on ? tri : cell * kCell;
  constexpr int NW = P1T ? 3 : 1;
  double phi[NO];
#pragma unroll
  for (int c = 0; c < NO; ++c) phi[c] = 0.0;
  __syncthreads();
  const int Q = WIDE ? d.far.Q : kQ;
  const size_t at = (size_t)sel * (WIDE ? d.far.nitems / d.far.ne * kWideItem : kQ);
#pragma unroll 1
  for (int first = 0; first < Q; first += kQ) {
    CellPoints p;
    load_points(d, sel, 1.0 / d.ball[cell].w, p, Q, first);
    double w[NW][kQ];
#pragma unroll
    for (int a = 0; a < kQ; ++a) {
      if constexpr (P1T) {
        const dq q = d.far.tgtw64[at + a];
        w[0][a] = q.x;
        w[1][a] = q.y;
        w[2][a] = q.z;
      } else {
        w[0][a] = first + a < Q ? d.far.tgt64[at + first + a].w : 0.0;
      }
    }
    each_harmonic<P>(tab, p, warp, [&](int n, int m, const double (&re)[kQ], const double (&im)[kQ]) {
      double hr[NW], hi[NW];
#pragma unroll
      for (int k = 0; k < NW; ++k) {
        hr[k] = hi[k] = 0.0;
#pragma unroll
        for (int a = 0; a < kQ; ++a) {
          hr[k] += w[k][a] * re[a];
          hi[k] += w[k][a] * im[a];
        }
      }
#pragma unroll
      for (int c = 0; c < NO; ++c) {
        const double2 l = s_loc[(P1T ? 0 : c) * kPairs + tree_pair(n, m)];
        phi[c] += l.x * hr[P1T ? c : 0] + l.y * hi[P1T ? c : 0];
      }
    });
  }
#pragma unroll
  for (int c = 0; c < NO; ++c) s_part[warp][c][lane] = phi[c];
  __syncthreads();
  if (warp == 0) {
    const size_t stride = (size_t)d.slot_off[d.ncells] * kCell;
    double* out = d.partial + d.first_col * stride + (size_t)(d.slot_off[cell + 1] - 1) * kCell + lane;
#pragma unroll
    for (int c = 0; c < NO; ++c) {
      double v = 0.0;
#pragma unroll
      for (int k = 0; k < kCellWarps; ++k) v += s_part[k][c][lane];
      out[c * stride] = v;
    }
  }
}

// ---------------------------------------------------------------------------
// Close cells: one warp per task, a lane per target triangle, the source cell
// staged in shared memory; every unordered pair of cells once, both orders
// (the transposed sums of a source cell go to its slot), a cell with itself
// in forward order.

template <typename T, int NSL, int ND>
constexpr int near_sources() { return sizeof(T) == 4 ? kCell : kCell / 2; }  // sources per reduction

template <typename T, int NSL, int ND>
constexpr size_t near_red_row()  // bytes of a lane's transposed sums, padded
{
  return ND > 0 ? 16 * (kCell / 2 + 1) : 8 * (kCell / 2 * NSL + 1);
}

template <typename T, int NSL, int ND>
constexpr size_t near_smem()
{
  return (size_t)kCell * kQ * kNrec * 4 * sizeof(T) + kCell * near_red_row<T, NSL, ND>();
}

// Sources of an entry of the close-pair lists.
struct NearSources {
  int cell, t0, ns;
  __device__ __forceinline__ NearSources(int x, int ne)
  {
    const int parts = x >> kTreePartsShift, part = x >> kTreePartShift & 7, n = kCell >> parts;
    cell = x & ((1 << kTreePartShift) - 1);
    t0 = cell * kCell + part * n;
    ns = max(0, min(n, ne - t0));
  }
};

template <typename T, int NSL, int ND>
__global__ void __launch_bounds__(32, 8)
    tree_near_kernel(const TreeDesc* __restrict__ descs, const int* __restrict__ off, int nmesh)
{
  using S = typename Slot<T>::type;
  constexpr bool F32 = sizeof(T) == 4;
  constexpr int NO = NSL + ND;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int4 s_vid[kCell];
  __shared__ dq s_nrm[ND ? kCell : 1];
  __shared__ S s_plane[ND ? kCell : 1];
  S* s_rec = reinterpret_cast<S*>(smem_raw);
  unsigned char* s_red = smem_raw + (size_t)kCell * kQ * kNrec * 4 * sizeof(T);
  const int lane = threadIdx.x;
  unsigned char* my_red = s_red + lane * near_red_row<T, NSL, ND>();
  int k = blockIdx.x;
  const TreeDesc& d = descs[tree_entry(off, nmesh, k)];
  const FarMeshDesc& md = d.far;
  if (md.active && *md.active == 0) return;
  const int4 task = d.tasks[k];
  const int ti = task.x * kCell + lane;
  const bool active = ti < md.ne;
  const int tsel = active ? ti : task.x * kCell;
  const dq ball = md.twarp[task.x];
  double cen[3], nrm[3] = {0.0, 0.0, 0.0}, pin = 0.0;
  {
    const dq c = md.tcent[tsel];
    cen[0] = c.x; cen[1] = c.y; cen[2] = c.z;
    if constexpr (ND > 0) {
      const dq n = md.snrm[tsel];
      nrm[0] = n.x; nrm[1] = n.y; nrm[2] = n.z;
      pin = n.w;
    }
  }
  const int4 tv = active ? md.tvid[tsel] : make_int4(-1, -1, -1, 0);
  const S* grec = reinterpret_cast<const S*>(md.rec);
  const size_t stride = (size_t)d.slot_off[d.ncells] * kCell;
  T hi[NO], lo[NO];
#pragma unroll
  for (int c = 0; c < NO; ++c) hi[c] = lo[c] = 0;

#pragma unroll 1
  for (int e = task.y; e < task.z; ++e) {
    const int2 en = d.entries[e];
    const NearSources src(en.x, md.ne);
    const int cell = src.cell, t0 = src.t0, ns = src.ns;
    {
      const S* g = grec + (size_t)t0 * kQ * kNrec;
      if constexpr (F32) {  // source-pair layout, as the symmetric kernel stages it
        constexpr int per = kQ * kNrec;
        const int nstage = ((ns + 1) >> 1) * per;
        for (int i = lane; i < nstage; i += 32) {
          const int p = i / per, rem = i - p * per;
          const float4 a = g[(size_t)(2 * p) * per + rem];
          float4 c;
          if (2 * p + 1 < ns) c = g[(size_t)(2 * p + 1) * per + rem];
          else c = rem % kNrec == 0 ? make_float4(0.f, 0.f, 0.f, 1.f) : make_float4(0.f, 0.f, 0.f, 0.f);
          s_rec[2 * i] = make_float4(a.x, c.x, a.y, c.y);
          s_rec[2 * i + 1] = make_float4(a.z, c.z, a.w, c.w);
        }
        if ((ns & 1) && lane == 0) {
          s_vid[ns] = make_int4(-1, -1, -1, 0);
          if constexpr (ND > 0) {
            s_nrm[ns] = dq{0.0, 0.0, 0.0, 0.0};
            s_plane[ns] = make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
      } else {
        for (int i = lane; i < ns * kQ * kNrec; i += 32) s_rec[i] = g[i];
      }
      if (lane < ns) {
        s_vid[lane] = md.svid[t0 + lane];
        if constexpr (ND > 0) {
          s_nrm[lane] = md.snrm[t0 + lane];
          if constexpr (F32) s_plane[lane] = md.splane32[t0 + lane];
          else s_plane[lane] = md.splane64[t0 + lane];
        }
      }
    }
    __syncwarp();
    const dq cc = md.ccent[cell];
    const double ddx = cc.x - ball.x, ddy = cc.y - ball.y, ddz = cc.z - ball.z;
    const double rr = kFarRatio * (cc.w + ball.w);
    const bool far = ddx * ddx + ddy * ddy + ddz * ddz > rr * rr;
    const T o[3] = {(T)(cc.x - cen[0]), (T)(cc.y - cen[1]), (T)(cc.z - cen[2])};
    T xs[kQ], ys[kQ], zs[kQ], q2[kQ], wq[kQ], part[NO];
#pragma unroll
    for (int a = 0; a < kQ; ++a) {
      S p;
      if constexpr (F32) p = md.tgt32[(size_t)tsel * kQ + a];
      else p = md.tgt64[(size_t)tsel * kQ + a];
      xs[a] = p.x - o[0]; ys[a] = p.y - o[1]; zs[a] = p.z - o[2];
      q2[a] = xs[a] * xs[a] + ys[a] * ys[a] + zs[a] * zs[a];
      wq[a] = p.w;
    }
    const double c3[3] = {cc.x, cc.y, cc.z};
#pragma unroll
    for (int c = 0; c < NO; ++c) part[c] = 0;
    if (cell == task.x) {
      T sl[NSL][kQ], dl[1][kQ];
#pragma unroll
      for (int a = 0; a < kQ; ++a) {
        dl[0][a] = 0;
#pragma unroll
        for (int c = 0; c < NSL; ++c) sl[c][a] = 0;
      }
      if (active) {
        if constexpr (F32)
          eval_cell_sp<kQ, kQ, NSL, ND, false>(s_rec, s_vid, s_nrm, s_plane, 0, ns, kQ, tv, xs, ys, zs, q2, o, cen, nrm,
                                               sl, dl);
        else
          eval_cell<T, kQ, kQ, NSL, ND, false>(s_rec, s_vid, s_nrm, s_plane, 0, ns, kQ, tv, xs, ys, zs, q2, o, cen, nrm,
                                               sl, dl);
      }
#pragma unroll
      for (int a = 0; a < kQ; ++a) {
#pragma unroll
        for (int c = 0; c < NSL; ++c) part[c] += wq[a] * sl[c][a];
        if constexpr (ND > 0) part[NSL] += wq[a] * dl[0][a];
      }
    } else {
      constexpr int kSrc = near_sources<T, NSL, ND>();
#pragma unroll 1
      for (int h = 0; h < ns; h += kSrc) {
        const int h1 = min(ns, h + kSrc);
        if (active) {
          // the target's strengths (SL + DL: s_a, c_a) and charges
          if constexpr (ND > 0) {
            T ca[kQ], cd[kQ], dl[kQ], slw = 0;
#pragma unroll
            for (int a = 0; a < kQ; ++a) {
              const S st = grec[((size_t)tsel * kQ + a) * kNrec + 1];
              cd[a] = st.x;
              ca[a] = st.y;
              dl[a] = 0;
            }
            if constexpr (F32) {
              float4* red = reinterpret_cast<float4*>(my_red);
              if (far) eval_cell_sym<true>(s_rec, s_vid, s_nrm, s_plane, h, h1, tv, xs, ys, zs, q2, ca, cd, wq, o, cen,
                                           nrm, c3, pin, slw, dl, red);
              else eval_cell_sym<false>(s_rec, s_vid, s_nrm, s_plane, h, h1, tv, xs, ys, zs, q2, ca, cd, wq, o, cen,
                                        nrm, c3, pin, slw, dl, red);
            } else {
              double2* red = reinterpret_cast<double2*>(my_red);
              if (far) eval_cell_sym64<true>(s_rec, s_vid, s_nrm, s_plane, h, h1, tv, xs, ys, zs, q2, ca, cd, wq, o,
                                             cen, nrm, c3, pin, slw, dl, red);
              else eval_cell_sym64<false>(s_rec, s_vid, s_nrm, s_plane, h, h1, tv, xs, ys, zs, q2, ca, cd, wq, o, cen,
                                          nrm, c3, pin, slw, dl, red);
            }
            part[0] += slw;
#pragma unroll
            for (int a = 0; a < kQ; ++a) part[NSL] += wq[a] * dl[a];
          } else {
            T cw[NSL][kQ], om[kQ], slw[NSL];
#pragma unroll
            for (int a = 0; a < kQ; ++a) {
              om[a] = wq[a] / wq[0];
              const S st = grec[((size_t)tsel * kQ + a) * kNrec + 1];
#pragma unroll
              for (int c = 0; c < NSL; ++c) cw[c][a] = wq[0] * comp(st, c);
            }
#pragma unroll
            for (int c = 0; c < NSL; ++c) slw[c] = 0;
            if constexpr (F32) {
              float2* red = reinterpret_cast<float2*>(my_red);
              if (far) eval_cell_sym_sl<NSL, true>(s_rec, s_vid, h, h1, tv, xs, ys, zs, q2, cw, om, wq, slw, red);
              else eval_cell_sym_sl<NSL, false>(s_rec, s_vid, h, h1, tv, xs, ys, zs, q2, cw, om, wq, slw, red);
            } else {
              double* red = reinterpret_cast<double*>(my_red);
              if (far) eval_cell_sym64_sl<NSL, true>(s_rec, s_vid, h, h1, tv, xs, ys, zs, q2, cw, om, wq, slw, red);
              else eval_cell_sym64_sl<NSL, false>(s_rec, s_vid, h, h1, tv, xs, ys, zs, q2, cw, om, wq, slw, red);
            }
#pragma unroll
            for (int c = 0; c < NSL; ++c) part[c] += slw[c];
          }
        } else {
          for (size_t i = 0; i < near_red_row<T, NSL, ND>() / 8; ++i) reinterpret_cast<double*>(my_red)[i] = 0.0;
        }
        __syncwarp();
        // lane l adds source triangle h + l over the 32 target lanes in order
        constexpr size_t row = near_red_row<T, NSL, ND>() / sizeof(T);
        const T* rf = reinterpret_cast<const T*>(s_red);
        if (h + lane < h1) {
#pragma unroll
          for (int c = 0; c < NO; ++c) {
            // FP32 sums of a triangle pair are interleaved
            int at;
            if constexpr (F32) at = ND > 0 ? (lane >> 1) * 4 + 2 * c + (lane & 1) : ((lane >> 1) * NSL + c) * 2 + (lane & 1);
            else at = lane * NO + c;
            T v0 = 0, v1 = 0, v2 = 0, v3 = 0;
#pragma unroll 4
            for (int t = 0; t < 32; t += 4) {
              v0 += rf[(t + 0) * row + at];
              v1 += rf[(t + 1) * row + at];
              v2 += rf[(t + 2) * row + at];
              v3 += rf[(t + 3) * row + at];
            }
            d.partial[c * stride + (size_t)en.y * kCell + (t0 - cell * kCell) + h + lane] = (double)((v0 + v1) + (v2 + v3));
          }
        }
        __syncwarp();
      }
    }
#pragma unroll
    for (int c = 0; c < NO; ++c) {
      if constexpr (F32) two_sum_add(hi[c], lo[c], part[c]);
      else hi[c] += part[c];
    }
    __syncwarp();
  }
#pragma unroll
  for (int c = 0; c < NO; ++c)
    d.partial[c * stride + (size_t)task.w * kCell + lane] = active ? (double)hi[c] + (double)lo[c] : 0.0;
}

// The same in forward order only: every cell against all its close cells (the
// full lists), for ND double-layer columns or (ND = 0) one single layer tested
// with the three hat functions. With four columns a pair costs 15 operations
// in either order; two symmetric passes of two columns, the most whose sums
// fit the registers, cost the same. P1 charges do not factor over a source's
// points, which the symmetric sums rely on.
template <typename T, int ND>
__global__ void __launch_bounds__(32, 8)
    tree_near_forward_kernel(const TreeDesc* __restrict__ descs, const int* __restrict__ off, int nmesh)
{
  using S = typename Slot<T>::type;
  constexpr bool F32 = sizeof(T) == 4;
  constexpr bool P1T = ND == 0;
  constexpr int NSL = P1T ? 1 : 0, NO = P1T ? 3 : ND, NDX = P1T ? 1 : ND;
  constexpr int NREC = rec_slots(NSL, ND);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int4 s_vid[kCell];
  __shared__ dq s_nrm[kCell];
  __shared__ S s_plane[kCell];
  S* s_rec = reinterpret_cast<S*>(smem_raw);
  const int lane = threadIdx.x;
  int k = blockIdx.x;
  const TreeDesc& d = descs[tree_entry(off, nmesh, k)];
  const FarMeshDesc& md = d.far;
  if (md.active && *md.active == 0) return;
  const int4 task = d.tasks[k];
  const int ti = task.x * kCell + lane;
  const bool active = ti < md.ne;
  const int tsel = active ? ti : task.x * kCell;
  const dq ball = md.twarp[task.x], cd = md.tcent[tsel], nd = md.tnrm[tsel];
  const double cen[3] = {cd.x, cd.y, cd.z}, nrm[3] = {nd.x, nd.y, nd.z};
  const int4 tv = active ? md.tvid[tsel] : make_int4(-1, -1, -1, 0);
  const S* grec = reinterpret_cast<const S*>(md.rec);
  T hi[NO], lo[NO];
#pragma unroll
  for (int c = 0; c < NO; ++c) hi[c] = lo[c] = 0;
#pragma unroll 1
  for (int e = task.y; e < task.z; ++e) {
    const NearSources src(d.entries[e].x, md.ne);
    const int cell = src.cell, t0 = src.t0, ns = src.ns;
    const S* g = grec + (size_t)t0 * kQ * NREC;
    if constexpr (F32) {  // source-pair layout
      constexpr int per = kQ * NREC;
      const int nstage = ((ns + 1) >> 1) * per;
      for (int i = lane; i < nstage; i += 32) {
        const int p = i / per, rem = i - p * per;
        const float4 a = g[(size_t)(2 * p) * per + rem];
        float4 c;
        if (2 * p + 1 < ns) c = g[(size_t)(2 * p + 1) * per + rem];
        else c = rem % NREC == 0 ? make_float4(0.f, 0.f, 0.f, 1.f) : make_float4(0.f, 0.f, 0.f, 0.f);
        s_rec[2 * i] = make_float4(a.x, c.x, a.y, c.y);
        s_rec[2 * i + 1] = make_float4(a.z, c.z, a.w, c.w);
      }
      if ((ns & 1) && lane == 0) {
        s_vid[ns] = make_int4(-1, -1, -1, 0);
        s_nrm[ns] = dq{0.0, 0.0, 0.0, 0.0};
        s_plane[ns] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    } else {
      for (int i = lane; i < ns * kQ * NREC; i += 32) s_rec[i] = g[i];
    }
    if (lane < ns) {
      s_vid[lane] = md.svid[t0 + lane];
      s_nrm[lane] = md.snrm[t0 + lane];
      if constexpr (F32) s_plane[lane] = md.splane32[t0 + lane];
      else s_plane[lane] = md.splane64[t0 + lane];
    }
    __syncwarp();
    if (active) {
      const dq cc = md.ccent[cell];
      const double ddx = cc.x - ball.x, ddy = cc.y - ball.y, ddz = cc.z - ball.z;
      const double rr = kFarRatio * (cc.w + ball.w);
      const bool far = ddx * ddx + ddy * ddy + ddz * ddz > rr * rr;
      const T o[3] = {(T)(cc.x - cen[0]), (T)(cc.y - cen[1]), (T)(cc.z - cen[2])};
      T xs[kQ], ys[kQ], zs[kQ], q2[kQ], wq[kQ], sl[1][kQ], dl[NDX][kQ];
#pragma unroll
      for (int a = 0; a < kQ; ++a) {
        S p;
        if constexpr (F32) p = md.tgt32[(size_t)tsel * kQ + a];
        else p = md.tgt64[(size_t)tsel * kQ + a];
        xs[a] = p.x - o[0]; ys[a] = p.y - o[1]; zs[a] = p.z - o[2];
        q2[a] = xs[a] * xs[a] + ys[a] * ys[a] + zs[a] * zs[a];
        wq[a] = p.w;
        sl[0][a] = 0;
#pragma unroll
        for (int c = 0; c < NDX; ++c) dl[c][a] = 0;
      }
      if constexpr (F32) {
        if (far) eval_cell_sp<kQ, kQ, NSL, ND, true>(s_rec, s_vid, s_nrm, s_plane, 0, ns, kQ, tv, xs, ys, zs, q2, o, cen, nrm, sl, dl);
        else eval_cell_sp<kQ, kQ, NSL, ND, false>(s_rec, s_vid, s_nrm, s_plane, 0, ns, kQ, tv, xs, ys, zs, q2, o, cen, nrm, sl, dl);
      } else {
        if (far) eval_cell<T, kQ, kQ, NSL, ND, true>(s_rec, s_vid, s_nrm, s_plane, 0, ns, kQ, tv, xs, ys, zs, q2, o, cen, nrm, sl, dl);
        else eval_cell<T, kQ, kQ, NSL, ND, false>(s_rec, s_vid, s_nrm, s_plane, 0, ns, kQ, tv, xs, ys, zs, q2, o, cen, nrm, sl, dl);
      }
#pragma unroll
      for (int c = 0; c < NO; ++c) {
        T part = 0;
#pragma unroll
        for (int a = 0; a < kQ; ++a) {
          if constexpr (P1T && F32) part += comp(md.tgtw32[(size_t)tsel * kQ + a], c) * sl[0][a];
          else if constexpr (P1T) part += comp(md.tgtw64[(size_t)tsel * kQ + a], c) * sl[0][a];
          else part += wq[a] * dl[c][a];
        }
        if constexpr (F32) two_sum_add(hi[c], lo[c], part);
        else hi[c] += part;
      }
    }
    __syncwarp();
  }
  const size_t stride = (size_t)d.slot_off[d.ncells] * kCell;
#pragma unroll
  for (int c = 0; c < NO; ++c)
    d.partial[c * stride + (size_t)task.w * kCell + lane] = active ? (double)hi[c] + (double)lo[c] : 0.0;
}

// The same for rules of more than 7 points, whose triangles are items of
// kWideItem target points (the last padded with zero weights): a lane runs its
// triangle's items one after the other against kWideTile staged sources, so
// that the FP64 records of a rule of 25 points leave 17 warps on an SM (4 with
// whole cells). Host apply of one operator, 8,192 triangles: rule of 16
// points FP64 12.44 -> 2.95 ms, mixed 5.95 -> 1.33; of 25, 38.3 -> 8.1 and
// 17.9 -> 3.7.
template <typename T, int NSL, int ND>
__global__ void __launch_bounds__(32)
    tree_near_wide_kernel(const TreeDesc* __restrict__ descs, const int* __restrict__ off, int nmesh)
{
  using S = typename Slot<T>::type;
  constexpr bool F32 = sizeof(T) == 4;
  constexpr int K = kWideItem, NO = NSL + ND, NSX = NSL > 0 ? NSL : 1, NDX = ND > 0 ? ND : 1;
  constexpr int NREC = rec_slots(NSL, ND);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int4 s_vid[kWideTile];
  __shared__ dq s_nrm[kWideTile];
  __shared__ S s_plane[kWideTile];
  S* s_rec = reinterpret_cast<S*>(smem_raw);
  const int lane = threadIdx.x;
  int k = blockIdx.x;
  const TreeDesc& d = descs[tree_entry(off, nmesh, k)];
  const FarMeshDesc& md = d.far;
  if (md.active && *md.active == 0) return;
  const int4 task = d.tasks[k];
  const int ti = task.x * kCell + lane;
  const bool active = ti < md.ne;
  const int tsel = active ? ti : task.x * kCell;
  const int Q = md.Q, nchunk = md.nitems / md.ne, per = Q * NREC;
  const size_t item0 = (size_t)tsel * nchunk;
  const dq ball = md.ccent[task.x], cd = md.tcent[item0], nd = md.tnrm[item0];
  const double cen[3] = {cd.x, cd.y, cd.z}, nrm[3] = {nd.x, nd.y, nd.z};
  const int4 tv = active ? md.tvid[item0] : make_int4(-1, -1, -1, 0);
  const S* grec = reinterpret_cast<const S*>(md.rec);
  T hi[NO], lo[NO];
#pragma unroll
  for (int c = 0; c < NO; ++c) hi[c] = lo[c] = 0;
#pragma unroll 1
  for (int e = task.y; e < task.z; ++e) {
    const NearSources src(d.entries[e].x, md.ne);
    const int cell = src.cell, end = src.t0 + src.ns;
    const dq cc = md.ccent[cell];
    const double ddx = cc.x - ball.x, ddy = cc.y - ball.y, ddz = cc.z - ball.z;
    const double rr = kFarRatio * (cc.w + ball.w);
    const bool far = ddx * ddx + ddy * ddy + ddz * ddz > rr * rr;
    const T o[3] = {(T)(cc.x - cen[0]), (T)(cc.y - cen[1]), (T)(cc.z - cen[2])};
#pragma unroll 1
    for (int t0 = src.t0; t0 < end; t0 += kWideTile) {
      const int ns = min(kWideTile, end - t0);
      const S* g = grec + (size_t)t0 * per;
      if constexpr (F32) {  // source-pair layout
        const int nstage = ((ns + 1) >> 1) * per;
        for (int i = lane; i < nstage; i += 32) {
          const int p = i / per, rem = i - p * per;
          const float4 a = g[(size_t)(2 * p) * per + rem];
          float4 c;
          if (2 * p + 1 < ns) c = g[(size_t)(2 * p + 1) * per + rem];
          else c = rem % NREC == 0 ? make_float4(0.f, 0.f, 0.f, 1.f) : make_float4(0.f, 0.f, 0.f, 0.f);
          s_rec[2 * i] = make_float4(a.x, c.x, a.y, c.y);
          s_rec[2 * i + 1] = make_float4(a.z, c.z, a.w, c.w);
        }
        if ((ns & 1) && lane == 0) {
          s_vid[ns] = make_int4(-1, -1, -1, 0);
          s_nrm[ns] = dq{0.0, 0.0, 0.0, 0.0};
          s_plane[ns] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
      } else {
        for (int i = lane; i < ns * per; i += 32) s_rec[i] = g[i];
      }
      if (lane < ns) {
        s_vid[lane] = md.svid[t0 + lane];
        s_nrm[lane] = md.snrm[t0 + lane];
        if constexpr (F32) s_plane[lane] = md.splane32[t0 + lane];
        else s_plane[lane] = md.splane64[t0 + lane];
      }
      __syncwarp();
      if (active) {
#pragma unroll 1
        for (int ch = 0; ch < nchunk; ++ch) {
          T xs[K], ys[K], zs[K], q2[K], wq[K], sl[NSX][K], dl[NDX][K];
#pragma unroll
          for (int a = 0; a < K; ++a) {
            S p;
            if constexpr (F32) p = md.tgt32[(item0 + ch) * K + a];
            else p = md.tgt64[(item0 + ch) * K + a];
            xs[a] = p.x - o[0]; ys[a] = p.y - o[1]; zs[a] = p.z - o[2];
            q2[a] = xs[a] * xs[a] + ys[a] * ys[a] + zs[a] * zs[a];
            wq[a] = p.w;
#pragma unroll
            for (int c = 0; c < NSX; ++c) sl[c][a] = 0;
#pragma unroll
            for (int c = 0; c < NDX; ++c) dl[c][a] = 0;
          }
          if constexpr (F32) {
            if (far) eval_cell_sp<K, 0, NSL, ND, true>(s_rec, s_vid, s_nrm, s_plane, 0, ns, Q, tv, xs, ys, zs, q2, o, cen, nrm, sl, dl);
            else eval_cell_sp<K, 0, NSL, ND, false>(s_rec, s_vid, s_nrm, s_plane, 0, ns, Q, tv, xs, ys, zs, q2, o, cen, nrm, sl, dl);
          } else {
            if (far) eval_cell<T, K, 0, NSL, ND, true>(s_rec, s_vid, s_nrm, s_plane, 0, ns, Q, tv, xs, ys, zs, q2, o, cen, nrm, sl, dl);
            else eval_cell<T, K, 0, NSL, ND, false>(s_rec, s_vid, s_nrm, s_plane, 0, ns, Q, tv, xs, ys, zs, q2, o, cen, nrm, sl, dl);
          }
#pragma unroll
          for (int c = 0; c < NO; ++c) {
            T part = 0;
#pragma unroll
            for (int a = 0; a < K; ++a) part += wq[a] * (c < NSL ? sl[c < NSL ? c : 0][a] : dl[c < NSL ? 0 : c - NSL][a]);
            if constexpr (F32) two_sum_add(hi[c], lo[c], part);
            else hi[c] += part;
          }
        }
      }
      __syncwarp();
    }
  }
  const size_t stride = (size_t)d.slot_off[d.ncells] * kCell;
#pragma unroll
  for (int c = 0; c < NO; ++c)
    d.partial[c * stride + (size_t)task.w * kCell + lane] = active ? (double)hi[c] + (double)lo[c] : 0.0;
}

// ---------------------------------------------------------------------------
// Tables (host, extended precision).

using ld = long double;

std::vector<std::vector<ld>> half_turns(int P)
{
  // Wigner's d^n_{m'm}(90 degrees), [n][(m' + n) (2n + 1) + m + n], by their
  // three-term recurrence in the degree n (stable upward) from n = max(|m|, |m'|)
  std::vector<std::vector<ld>> d(P + 1);
  for (int n = 0; n <= P; n++) d[n].assign((size_t)(2 * n + 1) * (2 * n + 1), 0.0L);
  auto binom = [](int n, int k) {
    ld v = 1.0L;
    for (int i = 1; i <= k; i++) v = v * (n - k + i) / i;
    return v;
  };
  for (int a = -P; a <= P; a++)
    for (int b = -P; b <= P; b++) {
      const int l0 = std::max(std::abs(a), std::abs(b));
      const ld half = std::pow(0.5L, l0);
      ld cur;
      if (a == l0) cur = std::sqrt(binom(2 * l0, l0 + b)) * half * ((l0 - b) & 1 ? -1 : 1);
      else if (a == -l0) cur = std::sqrt(binom(2 * l0, l0 + b)) * half;
      else if (b == l0) cur = std::sqrt(binom(2 * l0, l0 + a)) * half;
      else cur = std::sqrt(binom(2 * l0, l0 + a)) * half * ((l0 + a) & 1 ? -1 : 1);
      ld prev = 0.0L;
      for (int n = l0; n <= P; n++) {
        d[n][(size_t)(a + n) * (2 * n + 1) + b + n] = cur;
        ld next = 0.0L;
        if (n > 0)
          next = ((2 * n + 1) * (ld)(-a * b) * cur -
                  (n + 1) * std::sqrt((ld)(n * n - a * a) * (n * n - b * b)) * prev) /
                 (n * std::sqrt((ld)((n + 1) * (n + 1) - a * a) * ((n + 1) * (n + 1) - b * b)));
        prev = cur;
        cur = next;
      }
    }
  return d;
}

struct HostTables {
  std::vector<double> bmat, tmat[3];
  std::vector<int> pair;
  std::vector<double2> rec;
};

// Appends the fragment of tile t and step k of a block's matrix.
template <typename F>
void add_fragment(std::vector<double>& mat, int t, int k, F&& entry)
{
  for (int lane = 0; lane < 32; lane++)
    mat.push_back((double)entry(8 * t + (lane >> 3) + 4 * (lane >> 2 & 1), 4 * k + (lane & 3)));
}

HostTables make_tables(int P)
{
  HostTables h;
  const int els = 2 * ((P / 2 + 8) / 8), kt = (P + 4) / 4;
  const auto d = half_turns(P);
  for (int n = 0; n <= P; n++)
    for (int part = 0; part < 2; part++)
      for (int par = 0; par < 2; par++)
        for (int t = 0; t < els / 2; t++)
          for (int k = 0; k < els; k++)
            add_fragment(h.bmat, t, k, [&](int row, int col) -> ld {
              const int a = 2 * row + par, m = 2 * col + ((n + par + part) & 1);
              if (a > n || m > n || (part && (a == 0 || m == 0))) return 0.0L;
              const ld* r = &d[n][(size_t)(a + n) * (2 * n + 1)];
              if (m == 0) return r[n];
              const ld minus = (m & 1 ? -1 : 1) * r[n - m];
              return part ? r[n + m] - minus : r[n + m] + minus;
            });
  // along z; the powers of the step over the radii are applied to the
  // coefficients before and after
  std::vector<ld> fact(2 * P + 2, 1.0L);
  for (int k = 1; k < 2 * P + 2; k++) fact[k] = fact[k - 1] * k;
  auto norm = [&](int n, int m) { return std::sqrt(fact[n - m] * fact[n + m]); };
  for (int mode = 0; mode < 3; mode++)
    for (int m = 0; m <= P; m++)
      for (int t = 0; t < (kt + 1) / 2; t++)
        for (int s = 0; s < kt; s++)
          add_fragment(h.tmat[mode], t, s, [&](int row, int col) -> ld {
            const int n = m + row, k = m + col;
            if (n > P || k > P) return 0.0L;
            if (mode == kAcross) return ((n + m) & 1 ? -1 : 1) * fact[n + k] / (norm(n, m) * norm(k, m));
            if (mode == kUp) return k <= n ? norm(n, m) / (norm(k, m) * fact[n - k]) : 0.0L;
            return k >= n ? norm(k, m) / (norm(n, m) * fact[k - n]) : 0.0L;
          });
  h.rec.assign(tree_pairs(P), make_double2(0.0, 0.0));
  for (int n = 0; n <= P; n++)
    for (int m = 0; m <= n; m++) {
      h.pair.push_back(m | n << 8);
      if (n == m) {
        if (m > 0) h.rec[n * (n + 1) / 2 + m].x = -std::sqrt((2.0 * m - 1.0) / (2.0 * m));
      } else {
        const double q = (double)(n * n - m * m);
        h.rec[n * (n + 1) / 2 + m] =
            make_double2((2 * n - 1) / std::sqrt(q), std::sqrt(((n - 1.0) * (n - 1.0) - m * m) / q));
      }
    }
  return h;
}

// One set per device and order, made on first use and kept for the process
// (0.4 MB for both orders).
int tables_for(int device, int P, TreeTables* out)
{
  static std::mutex mu;
  static std::map<std::pair<int, int>, TreeTables> known;
  std::lock_guard<std::mutex> g(mu);
  const auto it = known.find({device, P});
  if (it != known.end()) {
    *out = it->second;
    return EB_OK;
  }
  const HostTables h = make_tables(P);
  std::vector<unsigned char> host;
  auto add = [&](const auto& v) {
    const size_t at = (host.size() + 15) & ~(size_t)15;
    host.resize(at + v.size() * sizeof(v[0]));
    std::memcpy(host.data() + at, v.data(), v.size() * sizeof(v[0]));
    return at;
  };
  const size_t at[] = {add(h.bmat), add(h.tmat[0]), add(h.tmat[1]), add(h.tmat[2]), add(h.pair), add(h.rec)};
  auto buf = std::make_unique<DevBuf>();
  EB_CHECK(buf->alloc(host.size()));
  EB_CHECK(copy_h2d(buf->p, host.data(), host.size()));
  const unsigned char* p = static_cast<const unsigned char*>(buf.release()->p);  // kept
  TreeTables t;
  t.bmat = reinterpret_cast<const double*>(p + at[0]);
  for (int k = 0; k < 3; k++) t.tmat[k] = reinterpret_cast<const double*>(p + at[1 + k]);
  t.pair = reinterpret_cast<const int*>(p + at[4]);
  t.rec = reinterpret_cast<const double2*>(p + at[5]);
  known[{device, P}] = t;
  *out = t;
  return EB_OK;
}

// ---------------------------------------------------------------------------
// Launches.

template <typename... Args>
cudaError_t start(void (*fn)(Args...), dim3 grid, int block, size_t smem, cudaStream_t st, Args... args)
{
  if (grid.x == 0) return cudaSuccess;
  if (smem > 32 * 1024) {  // per device: set on every launch (a host-side call)
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  fn<<<grid, block, smem, st>>>(args...);
  return cudaGetLastError();
}

template <int P, typename T, int NSL, int ND, bool P1 = false, bool WIDE = false>
int launch_all(const TreeDesc* d, const TreeGrid& g, const ApplyArgs& one, const ApplyArgs* many, const TreeTables& tab,
               const TreeSide& side, cudaStream_t st)
{
  constexpr int NC = NSL + ND;
  constexpr int MC = NC % 2 == 0 ? 2 : 1;  // columns of a CTA
  constexpr int PD = ND > 0 ? 1 : 0;       // double-layer columns of a multipole CTA
  using Mv = MoveShape<P, MC>;
  const dim3 b(Mv::kThreads);
  // close pairs beside the expansions; with nothing to run beside, on st itself
  cudaStream_t near = g.expansions ? side.st : st;
  if (g.expansions) {
    EB_CUDA(cudaEventRecord(side.fork, st));
    EB_CUDA(cudaStreamWaitEvent(side.st, side.fork, 0));
  }
  // a single double layer runs the SL+DL sums with zero charges (their records
  // hold zeros there; 1 of 9 or 14 operations), several the forward form
  if constexpr (P1)
    EB_CUDA(start(tree_near_forward_kernel<T, 0>, dim3(g.ntasks), 32, (size_t)kCell * kQ * rec_slots(1, 0) * 4 * sizeof(T),
                  near, d, g.tasks, g.nmesh));
  else if constexpr (WIDE)
    EB_CUDA(start(tree_near_wide_kernel<T, NSL, ND>, dim3(g.ntasks), 32,
                  (size_t)kWideTile * g.rule * rec_slots(NSL, ND) * 4 * sizeof(T), near, d, g.tasks, g.nmesh));
  else if constexpr (ND > 1)
    EB_CUDA(start(tree_near_forward_kernel<T, ND>, dim3(g.ntasks), 32, (size_t)kCell * kQ * rec_slots(0, ND) * 4 * sizeof(T),
                  near, d, g.tasks, g.nmesh));
  else
    EB_CUDA(start(tree_near_kernel<T, ND ? 1 : NSL, ND>, dim3(g.ntasks), 32, near_smem<T, ND ? 1 : NSL, ND>(), near, d,
                  g.tasks, g.nmesh));
  if (!g.expansions) return EB_OK;
  EB_CUDA(cudaEventRecord(side.join, side.st));
  if constexpr (P1)
    EB_CUDA(start(tree_p2m_kernel<P, 0, 1, kCharges>, dim3(g.ncells), 32 * kCellWarps, p2m_smem<P, 0, 1>(), st, d, g.cells,
                  g.nmesh, one, many, tab));
  else
    EB_CUDA(start(tree_p2m_kernel<P, NSL, PD, kApart, WIDE>, dim3(g.ncells, ND > 1 ? ND : 1), 32 * kCellWarps, p2m_smem<P, NSL, PD>(),
                  st, d, g.cells, g.nmesh, one, many, tab));
  for (int s = 0; s < kTreePasses; s++)
    EB_CUDA(start(tree_move_kernel<P, MC, kUp>, dim3(g.nup[s], NC / MC), b.x, Mv::smem(), st, d, g.up[s],
                  g.nmesh, s, tab));
  EB_CUDA(start(tree_move_kernel<P, MC, kAcross>, dim3(g.nm2l, NC / MC), b.x, Mv::smem(), st, d, g.m2l, g.nmesh,
                0, tab));
  EB_CUDA(start(tree_move_kernel<P, MC, kDown>, dim3(g.ncells, NC / MC), b.x, Mv::smem(), st, d, g.cells,
                g.nmesh, 0, tab));
  EB_CUDA(start(tree_l2p_kernel<P, NC, P1, WIDE>, dim3(g.ncells), 32 * kCellWarps, sizeof(double2) * NC * tree_pairs(P), st, d,
                g.cells, g.nmesh, tab));
  EB_CUDA(cudaStreamWaitEvent(st, side.join, 0));
  return EB_OK;
}

bool tree_variant(int nsl, int nd)
{
  if (nsl == kTreeP1) return nd == 0;
  return nd == 0 ? nsl == 1 || nsl == 3 || nsl == 4 : nsl == 0 ? nd == 1 || nd == 4 : nsl == 1 && nd == 1;
}

// ---------------------------------------------------------------------------
// Potentials at points off the surface: groups of at most 32 points, each from
// one cube of an octree along a Hilbert curve, take the separated nodes through
// local expansions of their own (the combination V t - W u as one column) and
// the close cells point by point: in FP64, in a mixed evaluation in FP32 unless
// the point lies within kPotNear radii of the cell (the rule of the direct
// evaluation).

constexpr int kGroup = 32;
constexpr int kCurveBits = 7;  // per dimension: two 11-bit passes of the host's radix sort

// Position of every point on the Hilbert curve through 2^kCurveBits cells per
// side (J. Skilling, "Programming the Hilbert curve", AIP Conf. Proc. 707
// (2004) 381); points outside or not finite go to the nearest side or 0.
__global__ void curve_kernel(int n, const double* __restrict__ pts, double ox, double oy, double oz, double inv,
                             unsigned* __restrict__ code)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double top = (1 << kCurveBits) - 1;
  const double o[3] = {ox, oy, oz};
  unsigned x[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double v = (pts[3 * (size_t)i + d] - o[d]) * inv;
    x[d] = v > 0.0 ? (unsigned)fmin(v, top) : 0u;
  }
#pragma unroll
  for (unsigned q = 1u << (kCurveBits - 1); q > 1; q >>= 1) {
    const unsigned p = q - 1;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (x[d] & q) {
        x[0] ^= p;
      } else {
        const unsigned t = (x[0] ^ x[d]) & p;
        x[0] ^= t;
        x[d] ^= t;
      }
    }
  }
  x[1] ^= x[0];
  x[2] ^= x[1];
  unsigned t = 0;
#pragma unroll
  for (unsigned q = 1u << (kCurveBits - 1); q > 1; q >>= 1)
    if (x[2] & q) t ^= q - 1;
  unsigned c = 0;
#pragma unroll
  for (int b = kCurveBits - 1; b >= 0; --b)
#pragma unroll
    for (int d = 0; d < 3; ++d) c = c << 1 | ((x[d] ^ t) >> b & 1);
  code[i] = c;
}

// Ball of every group (one warp each): box centre, largest distance, at least
// min_radius (points that coincide).
__global__ void group_ball_kernel(int ngroups, const int* __restrict__ gptr, const double* __restrict__ pts,
                                  const int* __restrict__ perm, double min_radius, dq* __restrict__ ball)
{
  const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (g >= ngroups) return;
  const int i = perm[min(gptr[g] + lane, gptr[g + 1] - 1)];
  const double p[3] = {pts[3 * (size_t)i], pts[3 * (size_t)i + 1], pts[3 * (size_t)i + 2]};
  double c[3], r2 = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    double lo = p[d], hi = p[d];
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    c[d] = 0.5 * (lo + hi);
    r2 += (p[d] - c[d]) * (p[d] - c[d]);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) r2 = fmax(r2, __shfl_xor_sync(0xffffffffu, r2, o));
  if (lane == 0) ball[g] = dq{c[0], c[1], c[2], fmax(sqrt(r2) * (1.0 + 1e-12), min_radius)};
}

constexpr int kPointCells = 4;  // close cells of a task
// Lists, expansions and partial sums of the groups evaluated at a time, kept by
// the mesh: only millions of points (150,000 groups in FP64), or groups that
// are close to hundreds of cells each, are cut. 6 million points, FP64: 2.3 GB
// at once, 0.4 GB in parts.
constexpr size_t kPointScratch = (size_t)1 << 30;
constexpr int kListWarps = 4;
// Nodes of a group still to be tested: 32 leave at a time and up to 64 children
// enter. Where these would reach the last kListReserve entries, one node leaves
// at a time, which adds at most one per level of the tree.
constexpr int kListStack = 1024, kListReserve = kTreePasses * kTreeLevelsPerPass + 1;
static_assert(kListReserve + 64 <= kListStack, "room for a step of 32 nodes");

// The tree against every group, a warp per group testing 32 nodes at a time:
// separated nodes that have a multipole and close cells, counted (FILL false)
// or written at the scanned offsets.
template <bool FILL>
__global__ void __launch_bounds__(32 * kListWarps)
    group_lists_kernel(int ngroups, int root, int ncells, double ratio, const dq* __restrict__ nodes,
                       const char* __restrict__ formed, const int2* __restrict__ child, const dq* __restrict__ ball,
                       int* __restrict__ far_ptr, int* __restrict__ near_ptr, int* __restrict__ task_ptr,
                       int* __restrict__ far, int* __restrict__ near)
{
  __shared__ int s_stack[kListWarps][kListStack];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = blockIdx.x * kListWarps + warp;
  if (g >= ngroups) return;
  int* stack = s_stack[warp];
  const unsigned below = (1u << lane) - 1;
  const dq b = ball[g];
  int nf = FILL ? far_ptr[g] : 0, nn = FILL ? near_ptr[g] : 0, top = 1;
  if (lane == 0) stack[0] = root;
  __syncwarp();
  while (top > 0) {
    const int take = min(min(32, top), max(1, kListStack - kListReserve - top));
    const int k = lane < take ? stack[top - 1 - lane] : -1;
    top -= take;
    __syncwarp();
    bool is_far = false, is_near = false;
    double d2 = 0.0, r = 0.0;
    if (k >= 0) {
      const dq x = nodes[k];
      const double dx = x.x - b.x, dy = x.y - b.y, dz = x.z - b.z;
      d2 = dx * dx + dy * dy + dz * dz;
      r = x.w;
      is_far = formed[k] && separated(r, b.w, d2, ratio);
      is_near = !is_far && k < ncells;
    }
    const bool split = k >= 0 && !is_far && !is_near;
    const unsigned mf = __ballot_sync(0xffffffffu, is_far), mn = __ballot_sync(0xffffffffu, is_near);
    const unsigned ms = __ballot_sync(0xffffffffu, split);
    if (FILL && is_far) far[nf + __popc(mf & below)] = (int)(degree_share(r, b.w, d2, ratio) << 24 | (unsigned)k);
    if (FILL && is_near) near[nn + __popc(mn & below)] = k;
    if (split) {
      const int2 c = child[k - ncells];
      const int at = top + 2 * __popc(ms & below);
      stack[at] = c.x;
      stack[at + 1] = c.y;
    }
    nf += __popc(mf);
    nn += __popc(mn);
    top += 2 * __popc(ms);
    __syncwarp();
  }
  if (!FILL && lane == 0) {
    far_ptr[g] = nf;
    near_ptr[g] = nn;
    task_ptr[g] = (nn + kPointCells - 1) / kPointCells;
  }
}

// Exclusive sums of a[0, n), b[0, n) and c[0, n) in place, totals at [n] and in
// total (one block). Sums past 2^31 wrap, the totals do not.
__global__ void __launch_bounds__(1024) scan_lists_kernel(int n, int* __restrict__ a, int* __restrict__ b,
                                                          int* __restrict__ c, long long* __restrict__ total)
{
  __shared__ int warps[3][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int* v[3] = {a, b, c};
  long long base[3] = {0, 0, 0};
  for (int i0 = 0; i0 < n; i0 += 1024) {
    const int i = i0 + threadIdx.x;
    int x[3], s[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      s[k] = x[k] = i < n ? v[k][i] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, s[k], o);
        if (lane >= o) s[k] += y;
      }
      if (lane == 31) warps[k][w] = s[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      long long before = base[k];
      for (int j = 0; j < 32; ++j) {
        if (j < w) before += warps[k][j];
        base[k] += warps[k][j];
      }
      if (i < n) v[k][i] = (int)(before + s[k] - x[k]);
    }
    __syncthreads();
  }
  if (threadIdx.x < 3) {
    v[threadIdx.x][n] = (int)base[threadIdx.x];
    total[threadIdx.x] = base[threadIdx.x];
  }
}

__global__ void iota_kernel(int n, int first, int* __restrict__ v)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) v[i] = first + i;
}

constexpr int kPointWarps = 4;

// One close cell's sum at a point in FP64, (xs, ys, zs) relative to its centre.
__device__ __forceinline__ double point_cell64(double xs, double ys, double zs, const dq* __restrict__ rec,
                                               const dq* __restrict__ plane, int ns)
{
  double part = 0.0;
#pragma unroll 1
  for (int s = 0; s < ns; ++s) {
    const dq pn = plane[s];
    const double d = xs * pn.x + (ys * pn.y + (zs * pn.z - pn.w));
    double sl = 0.0, acc = 0.0;
    const dq* r = rec + (size_t)s * kQ * kNrec;
#pragma unroll
    for (int k = 0; k < kQ; ++k) {
      const dq p0 = r[2 * k], p1 = r[2 * k + 1];
      const double ex = xs + 0.5 * p0.x, ey = ys + 0.5 * p0.y, ez = zs + 0.5 * p0.z;
      const double inv = rsq_f64(ex * ex + ey * ey + ez * ez);
      sl += p1.y * inv;
      acc += (inv * inv) * (p1.x * inv);
    }
    part += sl - d * acc;
  }
  return part;
}

// Close cells of the groups: a warp per task (kPointCells cells of one group),
// a lane per point, the cells staged one at a time (F32: FP32 records; the
// lanes close to the cell read the FP64 ones from global memory instead).
// part[task][lane] is the task's sum.
template <bool F32>
__global__ void __launch_bounds__(32 * kPointWarps)
    points_near_kernel(int ngroups, int ntasks, const int* __restrict__ gptr, const double* __restrict__ pts,
                       const int* __restrict__ perm, const int* __restrict__ task_ptr, const int* __restrict__ near_ptr,
                       const int* __restrict__ near, int ne, const float4* __restrict__ rec32,
                       const float4* __restrict__ plane32, const dq* __restrict__ rec64, const dq* __restrict__ plane64,
                       const dq* __restrict__ ccent, double* __restrict__ part_out)
{
  using S = typename std::conditional<F32, float4, dq>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ S s_plane[kPointWarps][kCell];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int task = blockIdx.x * kPointWarps + warp;
  if (task >= ntasks) return;  // warps are independent
  S* s_rec = reinterpret_cast<S*>(smem_raw) + (size_t)warp * kCell * kQ * kNrec;
  int g = 0;
  for (int hi = ngroups; hi - g > 1;) {  // task_ptr[g] <= task < task_ptr[hi]
    const int mid = (g + hi) >> 1;
    if (task_ptr[mid] <= task) g = mid;
    else hi = mid;
  }
  const int p = perm[min(gptr[g] + lane, gptr[g + 1] - 1)];
  const double px = pts[3 * (size_t)p], py = pts[3 * (size_t)p + 1], pz = pts[3 * (size_t)p + 2];
  const int e0 = near_ptr[g] + (task - task_ptr[g]) * kPointCells, e1 = min(near_ptr[g + 1], e0 + kPointCells);
  double sum = 0.0;
  float hi = 0.f, lo = 0.f;
#pragma unroll 1
  for (int e = e0; e < e1; ++e) {
    const int cell = near[e], t0 = cell * kCell, ns = min(kCell, ne - t0);
    const dq cc = ccent[cell];
    const double xs = px - cc.x, ys = py - cc.y, zs = pz - cc.z;
    const dq* r64 = rec64 + (size_t)t0 * kQ * kNrec;
    if constexpr (F32) {
      for (int i = lane; i < ns * kQ * kNrec; i += 32) s_rec[i] = rec32[(size_t)t0 * kQ * kNrec + i];
      if (lane < ns) s_plane[warp][lane] = plane32[t0 + lane];
      __syncwarp();
      if (xs * xs + ys * ys + zs * zs < kPotNear * kPotNear * cc.w * cc.w) {
        sum += point_cell64(xs, ys, zs, r64, plane64 + t0, ns);
      } else {
        const float X = (float)xs, Y = (float)ys, Z = (float)zs;
        float part = 0.f;
#pragma unroll 1
        for (int s = 0; s < ns; ++s) {
          const float4 pn = s_plane[warp][s];
          const float d = X * pn.x + (Y * pn.y + (Z * pn.z - pn.w));
          float sl = 0.f, acc = 0.f;
          const float4* r = s_rec + (size_t)s * kQ * kNrec;
#pragma unroll
          for (int k = 0; k < kQ; ++k) {
            const float4 p0 = r[2 * k], p1 = r[2 * k + 1];
            const float ex = X + 0.5f * p0.x, ey = Y + 0.5f * p0.y, ez = Z + 0.5f * p0.z;
            const float inv = rsq(ex * ex + ey * ey + ez * ez);
            sl += p1.y * inv;
            acc += (inv * inv) * (p1.x * inv);
          }
          part += sl - d * acc;
        }
        two_sum_add(hi, lo, part);
      }
    } else {
      for (int i = lane; i < ns * kQ * kNrec; i += 32) s_rec[i] = r64[i];
      if (lane < ns) s_plane[warp][lane] = plane64[t0 + lane];
      __syncwarp();
      sum += point_cell64(xs, ys, zs, s_rec, s_plane[warp], ns);
    }
    __syncwarp();
  }
  part_out[(size_t)task * 32 + lane] = sum + ((double)hi + (double)lo);
}

// Potentials of one group per warp, a lane per point: the local expansion and
// the sums of the group's tasks in order.
template <int P>
__global__ void __launch_bounds__(32 * kPointWarps)
    tree_points_kernel(int ngroups, const int* __restrict__ gptr, const double* __restrict__ pts,
                       const int* __restrict__ perm, const dq* __restrict__ ball, const double2* __restrict__ local,
                       const int* __restrict__ task_ptr, const double* __restrict__ part_in, TreeTables tab,
                       double* __restrict__ out)
{
  constexpr int kPairs = tree_pairs(P);
  __shared__ double2 s_all[kPointWarps][kPairs];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = blockIdx.x * kPointWarps + warp;
  if (g >= ngroups) return;  // warps are independent
  double2* s_loc = s_all[warp];
  for (int i = lane; i < kPairs; i += 32) s_loc[i] = local[(size_t)g * kPairs + i];
  const bool on = gptr[g] + lane < gptr[g + 1];
  const int p = perm[min(gptr[g] + lane, gptr[g + 1] - 1)];
  const dq b = ball[g];
  const double x = (pts[3 * (size_t)p] - b.x) / b.w, y = (pts[3 * (size_t)p + 1] - b.y) / b.w;
  const double z = (pts[3 * (size_t)p + 2] - b.z) / b.w, r2 = x * x + y * y + z * z;
  __syncwarp();
  double sum = 0.0;
  double dr = 1.0, di = 0.0;
#pragma unroll 1
  for (int m = 0; m <= P; ++m) {
    if (m > 0) {
      const double f = tab.rec[tree_pair(m, m)].x;
      const double t = f * (x * dr - y * di);
      di = f * (x * di + y * dr);
      dr = t;
    }
    double r1 = dr, i1 = di, r0 = 0.0, i0 = 0.0, part = 0.0;
#pragma unroll 4
    for (int d = m; d <= P; ++d) {
      const int q = tree_pair(d, m);
      if (d > m) {
        const double2 c = tab.rec[q];
        const double az = c.x * z, br = c.y * r2;
        const double tr = az * r1 - br * r0, ti = az * i1 - br * i0;
        r0 = r1;
        i0 = i1;
        r1 = tr;
        i1 = ti;
      }
      const double2 l = s_loc[q];
      part += l.x * r1 + l.y * i1;
    }
    sum += m > 0 ? 2.0 * part : part;
  }
  const int end = task_ptr[g + 1];
  for (int k = task_ptr[g]; k < end; ++k) sum += part_in[(size_t)k * 32 + lane];
  if (on) out[p] = sum * (0.25 / M_PI);
}

// The points of an evaluation that groups can hold, and the others: not finite,
// or so far out that squared distances overflow. One of those in a group would
// make its ball, and with it the expansion of every other point, infinite; the
// direct sums treat each point alone.
struct PointSet {
  std::vector<int> perm, apart;
  double lo[3], hi[3];  // box of perm
  PointSet(int n, const double* pts) : perm(n)
  {
    std::iota(perm.begin(), perm.end(), 0);
    if (box(pts)) return;
    perm.clear();
    for (int i = 0; i < n; i++) (inside(pts + 3 * (size_t)i) ? perm : apart).push_back(i);
    box(pts);
  }

 private:
  static bool inside(const double* p)
  {
    constexpr double kOutside = 1e150;
    return (std::fabs(p[0]) < kOutside) & (std::fabs(p[1]) < kOutside) & (std::fabs(p[2]) < kOutside);
  }
  // The box of perm; false when one of its points is outside.
  bool box(const double* pts)
  {
    double a[3] = {1e300, 1e300, 1e300}, b[3] = {-1e300, -1e300, -1e300};
    bool in = true;
    for (const int i : perm) {
      const double* p = pts + 3 * (size_t)i;
      in &= inside(p);
      for (int d = 0; d < 3; d++) {
        a[d] = p[d] < a[d] ? p[d] : a[d];
        b[d] = p[d] > b[d] ? p[d] : b[d];
      }
    }
    std::copy_n(a, 3, lo);
    std::copy_n(b, 3, hi);
    return in;
  }
};

__global__ void scatter_kernel(int n, const int* __restrict__ at, const double* __restrict__ v, double* __restrict__ out)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[at[i]] = v[i];
}

// Groups of an evaluation's points. An octree along a curve: its cubes are
// split while they hold more than kGroup points, small neighbours of one parent
// join. Two more rules keep points far out from spoiling it. Cubes of the last
// level that are still large against the mesh's cells (one far point stretches
// the first cube over all others) are divided anew from the box of their own
// points. And groups far from the mesh (2 / ratio radii of its root) whose
// points lie so far apart that not even the root is separated from them, which
// leaves all cells close, are halved until it is. 50,000 points around 81,920
// triangles, mixed / FP64 in ms (all inside: 2.3 / 7.9): one at a thousand times
// their distance 17.2 / 38.4 without the first rule, 2.95 / 8.1; distances over
// six decades 13.0 / 35.4 without both, 10.4 / 37.5 without the second, 4.9 / 10.9.
class PointGroups {
 public:
  // Sorts perm by its points' positions on the curve (code: those in a cube of side ext).
  PointGroups(const double* pts, const TreePlan& plan, double ratio, double ext, std::vector<unsigned>& code,
              std::vector<int>& perm)
      : pts_(pts), root_(plan.ball.back()), ratio_(ratio), code_(code), perm_(perm)
  {
    for (int c = 0; c < plan.ncells; c++) fine_ += plan.ball[c].w / plan.ncells;
    sort(0, (int)perm.size());
    split(0, (int)perm.size(), 0, ext);
  }
  std::vector<int> first;  // points of the groups in sorted order

 private:
  static constexpr int kBits = 11, kBins = 1 << kBits;
  static_assert(3 * kCurveBits <= 2 * kBits, "two passes cover the code");

  // Sorts perm[lo, hi) by code: two-pass radix sort, few points by comparison
  // (the bins of a pass cost as much as some 500 points).
  void sort(int lo, int hi)
  {
    const int n = hi - lo;
    if (n < kBins / 4) {
      std::sort(perm_.begin() + lo, perm_.begin() + hi,
                [this](int a, int b) { return code_[a] != code_[b] ? code_[a] < code_[b] : a < b; });
      return;
    }
    tmp_.resize(perm_.size());
    for (int pass = 0; pass < 2; pass++) {
      const int *from = pass ? tmp_.data() : perm_.data() + lo;
      int* to = pass ? perm_.data() + lo : tmp_.data();
      int cnt[kBins + 1] = {};
      for (int i = 0; i < n; i++) cnt[(code_[from[i]] >> (pass * kBits) & (kBins - 1)) + 1]++;
      for (int k = 0; k < kBins; k++) cnt[k + 1] += cnt[k];
      for (int i = 0; i < n; i++) to[cnt[code_[from[i]] >> (pass * kBits) & (kBins - 1)]++] = from[i];
    }
  }

  // Points lo .. hi of one cube of the given level, in a root cube of side ext.
  void split(int lo, int hi, int level, double ext)
  {
    if (hi - lo > kGroup && level == kCurveBits && divide(lo, hi, ext)) level = 0;
    const double side = ext / (1 << level);
    if (hi - lo <= kGroup || level == kCurveBits) {
      for (int i = lo; i < hi; i += kGroup) add(i, std::min(hi, i + kGroup), side);
      return;
    }
    const int shift = 3 * (kCurveBits - 1 - level);
    int start = lo;  // of the open group
    for (int i = lo; i < hi;) {
      const unsigned c = code_[perm_[i]] >> shift & 7;
      const int end = (int)(std::partition_point(perm_.begin() + i, perm_.begin() + hi,
                                                 [&](int p) { return (code_[p] >> shift & 7) == c; }) - perm_.begin());
      if (end - i > kGroup) {
        if (i > start) add(start, i, side);
        split(i, end, level + 1, ext);
        start = end;
      } else if (end - start > kGroup) {
        add(start, i, side);
        start = i;
      }
      i = end;
    }
    if (hi > start) add(start, hi, side);
  }

  // A group of points lo .. hi of a cube, or several.
  void add(int lo, int hi, double side)
  {
    if (hi - lo > 1 && (far_out(lo) || far_out(hi - 1)) && !separated_cube(lo, side)) {
      const Box box(*this, lo, hi);
      const double d2 = from_root(0.5 * (box.a[0] + box.b[0]), 0.5 * (box.a[1] + box.b[1]), 0.5 * (box.a[2] + box.b[2]));
      if (!separated(root_.w, std::sqrt(box.radius2()), d2, ratio_)) {
        int ax = 0;
        for (int d = 1; d < 3; d++)
          if (box.b[d] - box.a[d] > box.b[ax] - box.a[ax]) ax = d;
        const int mid = lo + (hi - lo) / 2;
        std::nth_element(perm_.begin() + lo, perm_.begin() + mid, perm_.begin() + hi, [&](int i, int j) {
          const double x = pts_[3 * (size_t)i + ax], y = pts_[3 * (size_t)j + ax];
          return x != y ? x < y : i < j;
        });
        add(lo, mid, side);
        add(mid, hi, side);
        return;
      }
    }
    first.push_back(lo);
  }

  // Whatever points a group holds of the cube that this one is from.
  bool separated_cube(int at, double side) const
  {
    const double* p = pts_ + 3 * (size_t)perm_[at];
    const double r = std::sqrt(0.75) * side, d = std::sqrt(from_root(p[0], p[1], p[2])) - 2.0 * r;
    return d > 0.0 && separated(root_.w, r, d * d, ratio_);
  }
  double from_root(double x, double y, double z) const
  {
    const double dx = x - root_.x, dy = y - root_.y, dz = z - root_.z;
    return dx * dx + dy * dy + dz * dz;
  }
  bool far_out(int at) const
  {
    const double* p = pts_ + 3 * (size_t)perm_[at];
    const double r = 2.0 / ratio_ * root_.w;
    return from_root(p[0], p[1], p[2]) > r * r;
  }

  struct Box {
    double a[3] = {1e300, 1e300, 1e300}, b[3] = {-1e300, -1e300, -1e300};
    Box(const PointGroups& g, int lo, int hi)
    {
      for (int i = lo; i < hi; i++)
        for (int d = 0; d < 3; d++) {
          a[d] = std::min(a[d], g.pts_[3 * (size_t)g.perm_[i] + d]);
          b[d] = std::max(b[d], g.pts_[3 * (size_t)g.perm_[i] + d]);
        }
    }
    double radius2() const
    {
      return 0.25 * ((b[0] - a[0]) * (b[0] - a[0]) + (b[1] - a[1]) * (b[1] - a[1]) + (b[2] - a[2]) * (b[2] - a[2]));
    }
  };

  // New codes in the box of points lo .. hi of a cube of the last level, and
  // their order (Morton: the host pays for it); false when the box is small.
  bool divide(int lo, int hi, double& ext)
  {
    if (std::sqrt(0.75) * ext / (1 << kCurveBits) <= fine_) return false;
    const Box box(*this, lo, hi);
    if (!(box.radius2() > fine_ * fine_)) return false;
    ext = std::max({box.b[0] - box.a[0], box.b[1] - box.a[1], box.b[2] - box.a[2]});
    const double inv = ((1 << kCurveBits) - 1e-6) / ext;
    for (int i = lo; i < hi; i++) {
      unsigned c = 0;
      for (int d = 0; d < 3; d++) {
        // bits of a coordinate three apart
        unsigned x = (unsigned)((pts_[3 * (size_t)perm_[i] + d] - box.a[d]) * inv);
        x = (x | x << 8) & 0x00f00fu;
        x = (x | x << 4) & 0x0c30c3u;
        x = (x | x << 2) & 0x249249u;
        c |= x << d;
      }
      code_[perm_[i]] = c;
    }
    sort(lo, hi);
    return true;
  }

  const double* pts_;
  const dq root_;
  const double ratio_;
  double fine_ = 0.0;  // mean radius of the cells
  std::vector<unsigned>& code_;
  std::vector<int>& perm_;
  std::vector<int> tmp_;
};

template <int P>
int evaluate_order(Mesh* m, int n, PointSet& set, const double* pts, const double* d_pts, const ApplyArgs& A,
                   const float4* rec32, const dq* rec64, double* d_out, cudaStream_t st)
{
  TreeMesh* t = m->tree.get();
  TreePoints& w = t->points;
  const TreePlan& plan = t->plan;
  constexpr int kPairs = tree_pairs(P);
  constexpr double ratio = P <= kTreeOrder32 ? kTreePointRatio32 : kTreePointRatio64;
  TreeTables tab;
  EB_CHECK(tables_for(m->device, P, &tab));
  // positions on the curve first: the host sorts them while the GPU forms the multipoles
  const double *lo = set.lo, *hi = set.hi;
  const double ext = std::max({hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2], 1e-300});
  EB_CHECK(w.code.alloc(sizeof(unsigned) * (size_t)n));
  EB_CHECK(w.perm.alloc(sizeof(int) * (size_t)n));
  EB_CHECK(w.multipole.alloc(sizeof(double2) * (size_t)plan.nnodes * kPairs));
  EB_CHECK(w.desc.alloc(2 * sizeof(TreeDesc)));
  curve_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, d_pts, lo[0], lo[1], lo[2], ((1 << kCurveBits) - 1e-6) / ext,
                                                w.code.as<unsigned>());
  EB_CUDA(cudaGetLastError());
  std::vector<unsigned> code(n);
  EB_CUDA(cudaMemcpyAsync(code.data(), w.code.p, sizeof(unsigned) * (size_t)n, cudaMemcpyDeviceToHost, st));
  EB_CUDA(cudaStreamSynchronize(st));  // the codes are here
  TreeDesc d[2];
  EB_CHECK(tree_desc(m, false, 1, 1, m->rec.p, w.multipole.p, nullptr, nullptr, &d[0]));
  TreeDesc* dd = w.desc.as<TreeDesc>();
  EB_CUDA(cudaMemcpyAsync(dd, &d[0], sizeof(TreeDesc), cudaMemcpyHostToDevice, st));
  using Mv = MoveShape<P, 1>;
  EB_CUDA(start(tree_p2m_kernel<P, 1, 1, kDiff>, dim3(plan.ncells), 32 * kCellWarps, p2m_smem<P, 1, 1>(), st,
                (const TreeDesc*)dd, (const int*)nullptr, 1, A, (const ApplyArgs*)nullptr, tab));
  for (int s = 0; s < kTreePasses; s++)
    EB_CUDA(start(tree_move_kernel<P, 1, kUp>, dim3(d[0].nup[s]), Mv::kThreads, Mv::smem(), st, (const TreeDesc*)dd,
                  (const int*)nullptr, 1, s, tab));
  std::vector<int>& perm = set.perm;
  const int npts = (int)perm.size();
  PointGroups groups(pts, plan, ratio, ext, code, perm);
  std::vector<int>& gptr = groups.first;
  const int ngroups = (int)gptr.size();
  gptr.push_back(npts);
  perm.insert(perm.end(), gptr.begin(), gptr.end());  // one copy
  EB_CHECK(w.perm.alloc(sizeof(int) * perm.size()));
  EB_CHECK(w.ball.alloc(sizeof(dq) * ((size_t)plan.nnodes + ngroups)));
  EB_CUDA(cudaMemcpyAsync(w.perm.p, perm.data(), sizeof(int) * perm.size(), cudaMemcpyHostToDevice, st));
  const int* d_perm = w.perm.as<int>();
  const int* d_gptr = d_perm + npts;
  // the groups as targets: nodes nnodes, nnodes + 1, ...
  dq* gball = w.ball.as<dq>() + plan.nnodes;
  EB_CUDA(cudaMemcpyAsync(w.ball.p, d[0].ball, sizeof(dq) * plan.nnodes, cudaMemcpyDeviceToDevice, st));
  const double root = plan.ball[plan.nnodes - 1].w;
  group_ball_kernel<<<(ngroups + 3) / 4, 128, 0, st>>>(ngroups, d_gptr, d_pts, d_perm, 1e-4 * root, gball);
  EB_CUDA(cudaGetLastError());
  // All groups at once where their lists, expansions and partial sums fit
  // kPointScratch, else as many at a time as fit whatever their lists hold.
  const size_t local_bytes = sizeof(double2) * kPairs, task_bytes = sizeof(double) * 32;
  const size_t most = local_bytes + 2 * sizeof(int) * (size_t)plan.ncells +
                      task_bytes * ((plan.ncells + kPointCells - 1) / kPointCells);
  const int slab = (int)std::max<size_t>(1, std::min<size_t>(ngroups, kPointScratch / most));
  for (int g0 = 0, step = ngroups; g0 < ngroups;) {
    const int ng = std::min(step, ngroups - g0);
    EB_CHECK(w.ptr.alloc(sizeof(long long) * 3 + sizeof(int) * 4 * ((size_t)ng + 1)));
    long long* d_total = w.ptr.as<long long>();
    int* far_ptr = reinterpret_cast<int*>(d_total + 3);
    int* near_ptr = far_ptr + ng + 1;
    int* task_ptr = near_ptr + ng + 1;
    int* ids = task_ptr + ng + 1;
    const int gb = (ng + kListWarps - 1) / kListWarps;
    group_lists_kernel<false><<<gb, 32 * kListWarps, 0, st>>>(ng, plan.nnodes - 1, plan.ncells, ratio, d[0].ball,
                                                              t->formed, t->children, gball + g0, far_ptr, near_ptr,
                                                              task_ptr, nullptr, nullptr);
    scan_lists_kernel<<<1, 1024, 0, st>>>(ng, far_ptr, near_ptr, task_ptr, d_total);
    iota_kernel<<<(ng + 255) / 256, 256, 0, st>>>(ng, plan.nnodes + g0, ids);
    EB_CUDA(cudaGetLastError());
    long long total[3];
    EB_CUDA(cudaMemcpyAsync(total, d_total, sizeof(total), cudaMemcpyDeviceToHost, st));
    EB_CUDA(cudaStreamSynchronize(st));
    if (step > slab && local_bytes * ng + sizeof(int) * (size_t)(total[0] + total[1]) +
                               task_bytes * (size_t)total[2] > kPointScratch) {
      step = slab;
      continue;
    }
    EB_CHECK(w.local.alloc(local_bytes * ng));
    EB_CHECK(w.part.alloc(task_bytes * (size_t)std::max(1ll, total[2])));
    EB_CHECK(w.far.alloc(sizeof(int) * (size_t)std::max(1ll, total[0])));
    EB_CHECK(w.near.alloc(sizeof(int) * (size_t)std::max(1ll, total[1])));
    d[1] = d[0];
    d[1].ball = w.ball.as<dq>();
    d[1].local = w.local.as<double2>() - (size_t)(plan.nnodes + g0) * kPairs;  // the first group's at its node
    d[1].m2l = TreeMovesDev{ids, far_ptr, w.far.as<int>()};
    EB_CUDA(cudaMemcpyAsync(dd + 1, &d[1], sizeof(TreeDesc), cudaMemcpyHostToDevice, st));
    group_lists_kernel<true><<<gb, 32 * kListWarps, 0, st>>>(ng, plan.nnodes - 1, plan.ncells, ratio, d[0].ball,
                                                             t->formed, t->children, gball + g0, far_ptr, near_ptr,
                                                             task_ptr, w.far.as<int>(), w.near.as<int>());
    EB_CUDA(cudaGetLastError());
    EB_CUDA(start(tree_move_kernel<P, 1, kAcross>, dim3(ng), Mv::kThreads, Mv::smem(), st, (const TreeDesc*)(dd + 1),
                  (const int*)nullptr, 1, 0, tab));
    constexpr bool F32 = P <= kTreeOrder32;
    const int ntasks = (int)total[2];
    EB_CUDA(start(points_near_kernel<F32>, dim3((ntasks + kPointWarps - 1) / kPointWarps), 32 * kPointWarps,
                  (size_t)kPointWarps * kCell * kQ * kNrec * (F32 ? sizeof(float4) : sizeof(dq)), st, ng, ntasks,
                  d_gptr + g0, d_pts, d_perm, (const int*)task_ptr, (const int*)near_ptr, (const int*)w.near.as<int>(),
                  m->h.ne, rec32, (const float4*)m->splane32.as<float4>(), rec64,
                  (const dq*)m->splane64.as<dq>(), (const dq*)m->ccent.as<dq>(), w.part.as<double>()));
    EB_CUDA(start(tree_points_kernel<P>, dim3((ng + kPointWarps - 1) / kPointWarps), 32 * kPointWarps, 0, st, ng,
                  d_gptr + g0, d_pts, d_perm, (const dq*)(gball + g0), (const double2*)w.local.as<double2>(),
                  (const int*)task_ptr, (const double*)w.part.as<double>(), tab, d_out));
    g0 += ng;
  }
  EB_CUDA(cudaStreamSynchronize(st));  // perm and d are read by the copies
  return EB_OK;
}

}  // namespace

int tree_launch(bool fp32, int nsl, int nd, const TreeDesc* d, const TreeGrid& g, const ApplyArgs& one,
                const ApplyArgs* many, int device, const TreeSide& side, cudaStream_t st)
{
  TreeTables tab = {};
  if (g.expansions) EB_CHECK(tables_for(device, fp32 ? kTreeOrder32 : kTreeOrder64, &tab));
  if (nsl == kTreeP1 && nd == 0)
    return fp32 ? launch_all<kTreeOrder32, float, 1, 0, true>(d, g, one, many, tab, side, st)
                : launch_all<kTreeOrder64, double, 1, 0, true>(d, g, one, many, tab, side, st);
#define EB_TREE(NSL, ND)                                                                        \
  if (nsl == NSL && nd == ND)                                                                   \
    return fp32 ? launch_all<kTreeOrder32, float, NSL, ND>(d, g, one, many, tab, side, st)            \
                : launch_all<kTreeOrder64, double, NSL, ND>(d, g, one, many, tab, side, st);
#define EB_TREE_WIDE(NSL, ND)                                                                         \
  if (g.rule > kQ && nsl == NSL && nd == ND)                                                          \
    return fp32 ? launch_all<kTreeOrder32, float, NSL, ND, false, true>(d, g, one, many, tab, side, st)  \
                : launch_all<kTreeOrder64, double, NSL, ND, false, true>(d, g, one, many, tab, side, st);
  EB_TREE_WIDE(1, 1)
  EB_TREE_WIDE(1, 0)
  EB_TREE_WIDE(0, 1)
#undef EB_TREE_WIDE
  EB_TREE(1, 1)
  EB_TREE(1, 0)
  EB_TREE(3, 0)
  EB_TREE(4, 0)
  EB_TREE(0, 1)
  EB_TREE(0, 4)
#undef EB_TREE
  return set_error(EB_ERR_INVALID, "no tree far field for this operator combination");
}

// Rules of 8 points and more take the tree in the single variants, on meshes
// that have expansions: their close pairs run in forward order only, which
// gains nothing where every pair is close.
static bool wide_rule(const HostMesh& h) { return h.K == kWideItem; }

void tree_prepare(Mesh* m)
{
  const HostMesh& h = m->h;
  m->tree.reset();
  const bool wide = wide_rule(h);
  if (!wide && (h.Q != kSymRule || h.K != kSymRule || h.nchunk != 1)) return;
  m->tree = std::make_shared<TreeMesh>();
  m->tree->usable = make_tree_plan(h, &m->tree->plan) && !(wide && m->tree->plan.all_close);
}

bool tree_eligible(const Mesh* m, int nsl, int nd, bool fp32)
{
  if (nd > 1 && m->tree && m->tree->plan.all_close && m->h.ncells > (fp32 ? kTreeForwardCells32 : kTreeForwardCells64))
    return false;
  return m->plan.engine == 4 && m->tree && m->tree->usable && tree_variant(nsl, nd) &&
         (!wide_rule(m->h) || (nsl <= 1 && nd <= 1)) && tree_partial_bytes(m, nsl, nd) <= kTreeMaxSlotBytes;
}

// With t->lists_lock held, as upload_forward.
static int upload_lists(TreeMesh* t)
{
  if (t->lists_ready) return EB_OK;
  const TreePlan& p = t->plan;
  std::vector<unsigned char> host;
  auto add = [&](const auto& v) {
    const size_t at = (host.size() + 15) & ~(size_t)15;
    host.resize(at + std::max<size_t>(1, v.size()) * sizeof(v[0]));
    if (!v.empty()) std::memcpy(host.data() + at, v.data(), v.size() * sizeof(v[0]));
    return at;
  };
  const size_t child = add(p.child), formed = add(p.formed), ball = add(p.ball), has = add(p.has_local), tasks = add(p.sym.tasks), entries = add(p.sym.entries),
               slots = add(p.sym.slot_off);
  struct At {
    size_t tgt, ptr, src;
  };
  auto moves = [&](const TreeMoves& m) { return At{add(m.tgt), add(m.ptr), add(m.src)}; };
  At up[kTreePasses];
  for (int s = 0; s < kTreePasses; s++) up[s] = moves(p.up[s]);
  const At m2l = moves(p.m2l), down = moves(p.down);
  EB_CHECK(t->lists.alloc(host.size()));
  EB_CHECK(copy_h2d(t->lists.p, host.data(), host.size()));
  const unsigned char* q = static_cast<const unsigned char*>(t->lists.p);
  auto dev = [&](const At& a) {
    return TreeMovesDev{reinterpret_cast<const int*>(q + a.tgt), reinterpret_cast<const int*>(q + a.ptr),
                        reinterpret_cast<const int*>(q + a.src)};
  };
  TreeDesc& d = t->base;
  t->children = reinterpret_cast<const int2*>(q + child);
  t->formed = reinterpret_cast<const char*>(q + formed);
  d.ball = reinterpret_cast<const dq*>(q + ball);
  d.has_local = reinterpret_cast<const char*>(q + has);
  d.tasks = reinterpret_cast<const int4*>(q + tasks);
  d.entries = reinterpret_cast<const int2*>(q + entries);
  d.slot_off = reinterpret_cast<const int*>(q + slots);
  for (int s = 0; s < kTreePasses; s++) {
    d.up[s] = dev(up[s]);
    d.nup[s] = (int)p.up[s].tgt.size();
  }
  d.m2l = dev(m2l);
  d.down = dev(down);
  d.nnodes = p.nnodes;
  d.ncells = p.ncells;
  d.ntasks = (int)p.sym.tasks.size();
  d.nm2l = (int)p.m2l.tgt.size();
  t->lists_ready = true;
  return EB_OK;
}

int TreeSide::create()
{
  if (st) return EB_OK;
  int least = 0, greatest = 0;
  EB_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
  EB_CUDA(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
  EB_CUDA(cudaEventCreateWithFlags(&join, cudaEventDisableTiming));
  EB_CUDA(cudaStreamCreateWithPriority(&st, cudaStreamNonBlocking, least));
  return EB_OK;
}

TreeSide::~TreeSide()
{
  if (st) cudaStreamDestroy(st);
  if (fork) cudaEventDestroy(fork);
  if (join) cudaEventDestroy(join);
}

// Close pairs of a variant in both orders at once, or forward only.
static bool tree_forward(const Mesh* m, int nsl, int nd) { return nd > 1 || nsl == kTreeP1 || wide_rule(m->h); }
// Columns of its expansions and of its slots (a double layer alone in both
// orders leaves the single layer's column unused).
static int moved_columns(int nsl, int nd) { return nsl == kTreeP1 ? 1 : nsl + nd; }
static int unused_columns(const Mesh* m, int nsl, int nd) { return nsl == 0 && nd == 1 && !wide_rule(m->h) ? 1 : 0; }
static int slot_columns(const Mesh* m, int nsl, int nd)
{
  return nsl == kTreeP1 ? 3 : nsl + nd + unused_columns(m, nsl, nd);
}

long long tree_far_slots(const Mesh* m, int nsl, int nd)
{
  const TreePlan& p = m->tree->plan;
  return (long long)(tree_forward(m, nsl, nd) ? p.forward_slots : p.sym.slot_off.back()) * kCell;
}

static int upload_forward(TreeMesh* t)
{
  if (t->fwd_ready) return EB_OK;
  TreeNear& f = t->fwd;
  f = TreeNear();
  make_near_lists(t->plan, false, &f);
  const size_t a = f.tasks.size() * sizeof(int4), b = f.entries.size() * sizeof(int2), c = f.slot_off.size() * sizeof(int);
  std::vector<unsigned char> host(a + b + c);
  std::memcpy(host.data(), f.tasks.data(), a);
  std::memcpy(host.data() + a, f.entries.data(), b);
  std::memcpy(host.data() + a + b, f.slot_off.data(), c);
  EB_CHECK(t->fwd_lists.alloc(host.size()));
  EB_CHECK(copy_h2d(t->fwd_lists.p, host.data(), host.size()));
  t->fwd_ready = true;
  return EB_OK;
}

int tree_tables(bool fp32, int device)
{
  TreeTables tab;
  return tables_for(device, fp32 ? kTreeOrder32 : kTreeOrder64, &tab);
}

size_t tree_expansion_bytes(const Mesh* m, int order, int cols)
{
  return m->tree->plan.all_close ? 0 : sizeof(double2) * (size_t)cols * m->tree->plan.nnodes * tree_pairs(order);
}

size_t tree_partial_bytes(const Mesh* m, int nsl, int nd)
{
  return sizeof(double) * (size_t)slot_columns(m, nsl, nd) * tree_far_slots(m, nsl, nd);
}

int tree_desc(Mesh* m, bool fp32, int nsl, int nd, void* rec, void* multipole, void* local, double* partial,
              TreeDesc* out)
{
  TreeMesh* t = m->tree.get();
  std::lock_guard<std::mutex> g(t->lists_lock);
  EB_CHECK(upload_lists(t));
  TreeDesc d = t->base;
  if (tree_forward(m, nsl, nd)) {
    EB_CHECK(upload_forward(t));
    d.tasks = t->fwd_lists.as<int4>();
    d.entries = reinterpret_cast<const int2*>(d.tasks + t->fwd.tasks.size());
    d.slot_off = reinterpret_cast<const int*>(d.entries + t->fwd.entries.size());
    d.ntasks = (int)t->fwd.tasks.size();
  }
  d.far = mesh_far_desc(m, fp32, nsl == kTreeP1 ? 1 : nsl, nd, rec, partial);
  d.pos = m->pos64.as<dq>();
  d.multipole = static_cast<double2*>(multipole);
  d.local = static_cast<double2*>(local);
  d.partial = partial;
  d.first_col = unused_columns(m, nsl, nd);
  *out = d;
  return EB_OK;
}

void tree_finalize_args(const Mesh* m, int nsl, int nd, const TreeDesc& d, ApplyArgs* A)
{
  A->partial = d.partial + (size_t)d.first_col * tree_far_slots(m, nsl, nd);
  A->slot_off = d.slot_off;
}

bool tree_points_eligible(const Mesh* m, bool fp32, int npts)
{
  const double n = npts, ne = m->h.ne;
  const double least = fp32 ? kTreePointPairs32 + kTreePointTriangles32 * ne + kTreePointPoints32 * n
                            : kTreePointPairs64 + kTreePointTriangles64 * ne + kTreePointPoints64 * n;
  return m->plan.engine == 4 && m->tree && m->tree->usable && !m->tree->plan.all_close && !wide_rule(m->h) && n * ne >= least;
}

// Direct sums at the points that are set apart.
static int evaluate_apart(Mesh* m, bool fp32, const std::vector<int>& apart, const double* pts, const double* d_t,
                          const double* d_u, double* d_out, cudaStream_t st)
{
  const size_t n = apart.size();
  std::vector<double> x(3 * n);
  for (size_t i = 0; i < n; i++) std::copy_n(pts + 3 * (size_t)apart[i], 3, &x[3 * i]);
  DevBuf& w = m->tree->points.apart;
  EB_CHECK(w.alloc(n * (4 * sizeof(double) + sizeof(int))));
  double *d_x = w.as<double>(), *d_v = d_x + 3 * n;
  int* d_at = reinterpret_cast<int*>(d_v + n);
  EB_CUDA(cudaMemcpyAsync(d_x, x.data(), sizeof(double) * 3 * n, cudaMemcpyHostToDevice, st));
  EB_CUDA(cudaMemcpyAsync(d_at, apart.data(), sizeof(int) * n, cudaMemcpyHostToDevice, st));
  EB_CHECK(mesh_evaluate_potential(m, fp32 ? EB_PREC_MIXED : EB_PREC_FP64, (int)n, d_x, d_t, d_u, d_v, st));
  scatter_kernel<<<((int)n + 255) / 256, 256, 0, st>>>((int)n, d_at, d_v, d_out);
  EB_CUDA(cudaGetLastError());
  EB_CUDA(cudaStreamSynchronize(st));  // x is read by the copy
  return EB_OK;
}

int tree_evaluate(Mesh* m, bool fp32, int npts, const double* pts, const double* d_pts, const double* d_t,
                  const double* d_u, double* d_out, cudaStream_t st)
{
  PointSet set(npts, pts);
  if (!set.perm.empty()) {
    // FP64 records in either precision (the cells closest to a point), FP32 ones beside them
    DevBuf& rec = m->pot_rec64;
    EB_CHECK(rec.alloc((size_t)m->h.ne * m->h.Q * rec_slots(1, 1) * sizeof(dq)));
    const ApplyArgs A = mesh_apply_args(m, false, rec.p, nullptr, d_t, m->h.ne, d_u, nullptr, m->h.ne, nullptr);
    EB_CUDA(prep_launch(false, 1, 1, A, st));
    if (fp32) {
      EB_CHECK(ensure_apply_scratch(m, true));
      const ApplyArgs A32 = mesh_apply_args(m, true, m->rec.p, nullptr, d_t, m->h.ne, d_u, nullptr, m->h.ne, nullptr);
      EB_CUDA(prep_launch(true, 1, 1, A32, st));
      EB_CHECK(evaluate_order<kTreeOrder32>(m, npts, set, pts, d_pts, A, m->rec.as<float4>(), rec.as<dq>(), d_out, st));
    } else {
      EB_CHECK(evaluate_order<kTreeOrder64>(m, npts, set, pts, d_pts, A, nullptr, rec.as<dq>(), d_out, st));
    }
  }
  return set.apart.empty() ? EB_OK : evaluate_apart(m, fp32, set.apart, pts, d_t, d_u, d_out, st);
}

size_t tree_bytes(const Mesh* m)
{
  if (!m->tree) return 0;
  size_t b = 0;
  {
    std::lock_guard<std::mutex> g(m->tree->lists_lock);
    b += m->tree->lists.bytes + m->tree->fwd_lists.bytes;
  }
  for (const auto& s : m->tree->scratch)
    b += s.second->multipole.bytes + s.second->local.bytes + s.second->partial.bytes + s.second->desc.bytes;
  const TreePoints& w = m->tree->points;
  for (const DevBuf* d : {&w.code, &w.perm, &w.multipole, &w.local, &w.ball, &w.ptr, &w.far, &w.near, &w.part, &w.desc,
                          &w.apart})
    b += d->bytes;
  return b;
}

void tree_release_scratch(Mesh* m)
{
  if (!m->tree) return;
  m->tree->scratch.clear();
  TreePoints& w = m->tree->points;
  for (DevBuf* d : {&w.code, &w.perm, &w.multipole, &w.local, &w.ball, &w.ptr, &w.far, &w.near, &w.part, &w.desc,
                    &w.apart})
    d->release();
}

int tree_far_apply(Mesh* m, bool fp32, int nsl, int nd, ApplyArgs* A, cudaStream_t st)
{
  TreeMesh* t = m->tree.get();
  if (!t->plan.all_close) EB_CHECK(t->side.create());
  std::unique_ptr<TreeScratch>& sc = t->scratch[(fp32 ? 64 : 0) + nsl * 5 + nd];
  if (!sc) {
    auto s = std::make_unique<TreeScratch>();
    const size_t bytes = tree_expansion_bytes(m, fp32 ? kTreeOrder32 : kTreeOrder64, moved_columns(nsl, nd));
    if (bytes) {
      EB_CHECK(s->multipole.alloc(bytes));
      EB_CHECK(s->local.alloc(bytes));
    }
    EB_CHECK(s->partial.alloc(tree_partial_bytes(m, nsl, nd)));
    EB_CHECK(tree_desc(m, fp32, nsl, nd, m->rec.p, s->multipole.p, s->local.p, s->partial.as<double>(), &s->host));
    EB_CHECK(s->desc.alloc(sizeof(TreeDesc)));
    EB_CHECK(copy_h2d(s->desc.p, &s->host, sizeof(TreeDesc)));
    sc = std::move(s);
  }
  const TreeDesc& d = sc->host;
  tree_finalize_args(m, nsl, nd, d, A);
  TreeGrid g;
  g.rule = m->h.Q;
  g.ncells = d.ncells;
  g.nm2l = d.nm2l;
  g.ntasks = d.ntasks;
  g.expansions = !t->plan.all_close;
  std::copy_n(d.nup, kTreePasses, g.nup);
  if (m->profile) EB_CUDA(cudaEventRecord(m->ev0, st));
  return tree_launch(fp32, nsl, nd, sc->desc.as<TreeDesc>(), g, *A, nullptr, m->device, t->side, st);
}

}  // namespace eb
