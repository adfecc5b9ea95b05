// Device-side evaluation of one source cell against one target triangle, both
// orders of every pair (7-point rule): the inner loops of the symmetric far
// field (farfield_sym.cu, which derives the form) and of the near cells of the
// tree far field (farfield_tree.cu).
#pragma once

#include <cuda_runtime.h>

#include "farfield.cuh"
#include "farfield_eval.cuh"
#include "farfield_sym.h"

// Source-point unroll of the symmetric pair loop (0: full).
#ifndef EB_SYM_UNROLL_B
#define EB_SYM_UNROLL_B 0
#endif
// Source-point unroll of the FP64 symmetric loop (0: full).
#ifndef EB_SYM_UNROLL_B64
#define EB_SYM_UNROLL_B64 0
#endif

namespace eb {

constexpr int kQ = kSymRule;
constexpr int kUnrollB = EB_SYM_UNROLL_B > 0 ? EB_SYM_UNROLL_B : kQ;
constexpr int kUnrollB64 = EB_SYM_UNROLL_B64 > 0 ? EB_SYM_UNROLL_B64 : kQ;
constexpr int kNrec = 2;  // rec_slots(1, 1): (-2y, |y|^2), (s, c, J t, 0)

__device__ __forceinline__ float2 bcast(float v) { return make_float2(v, v); }

// One target triangle (kQ points, relative to the cell centre) against the
// source triangles [s0, s1) of one cell of the staged pair-interleaved tile,
// both orders of every pair. Forward sums: the single layer as one sum
// already weighted by the target points' rule weights (slw), the double
// layer per target point (dl, as eval_cell_sp); the transposed sums of
// source triangles s, s+1 go to red[s / 2] as (SL s, SL s+1, DL s, DL s+1),
// weighted by the source points' rule weights w_b (the finalize multiplies a
// row by J / 4 pi).
//
// Single layer: both charges factor as c = w J t, so one sum per target
// point, R_a = sum_b w_b / r_ab, serves both rows: row i gets J_j t_j
// sum_a w_a R_a, row j gets sum_a c_a R_a (1 FMA per pair instead of 2).
//
// Far cells: expanded |x - y|^2 and e_i(y) = (y - c).n_i + (c - P0_i).n_i;
// other cells: direct differences, a 1e-24 floor and, per lane, e_i(y) =
// (y - c).(n_i - n_j) + (P0_j.n_j - P0_i.n_i) + c.(n_i - n_j) (exact for y in
// the plane of j; the normal difference keeps e small and accurate for
// nearly coplanar neighbours); lanes whose triangle shares a vertex with the
// target get zero strengths and zero transposed sums.
template <bool FAR>
__device__ __forceinline__ void eval_cell_sym(const float4* __restrict__ srec, const int4* __restrict__ svid,
                                              const dq* __restrict__ snrm, const float4* __restrict__ splane, int s0,
                                              int s1, int4 tv, const float (&x)[kQ], const float (&y)[kQ],
                                              const float (&z)[kQ], const float (&q2)[kQ], const float (&ca)[kQ],
                                              const float (&cd)[kQ], const float (&wq)[kQ], const float (&o)[3],
                                              const double (&cen)[3], const double (&nrm)[3],
                                              const double (&cc)[3], double pin, float& slw, float (&dl)[kQ],
                                              float4* __restrict__ red)
{
  float2 X[kQ], Y[kQ], Z[kQ], W[kQ], DLp[kQ];
  float2 SLW = make_float2(0.f, 0.f);
#pragma unroll
  for (int a = 0; a < kQ; ++a) {
    X[a] = bcast(x[a]);
    Y[a] = bcast(y[a]);
    Z[a] = bcast(z[a]);
    W[a] = bcast(q2[a]);
    DLp[a] = make_float2(0.f, 0.f);
  }
  const float2 half2 = bcast(0.5f);
  const float2 eps2 = bcast(1e-24f);
  // plane of the target triangle seen from the cell centre (far cells)
  float2 EX, EY, EZ, EW;
  if constexpr (FAR) {
    EX = bcast(-0.5f * (float)nrm[0]);
    EY = bcast(-0.5f * (float)nrm[1]);
    EZ = bcast(-0.5f * (float)nrm[2]);
    EW = bcast((float)(cc[0] * nrm[0] + cc[1] * nrm[1] + cc[2] * nrm[2] - pin));
  }
#pragma unroll 1
  for (int s = s0; s < s1; s += 2) {
    float2 keep = make_float2(1.f, 1.f);
    if constexpr (!FAR) {
      const bool m0 = shares_vertex(tv, svid[s]), m1 = shares_vertex(tv, svid[s + 1]);
      if (m0 && m1) {
        red[s >> 1] = make_float4(0.f, 0.f, 0.f, 0.f);
        continue;
      }
      keep = make_float2(m0 ? 0.f : 1.f, m1 ? 0.f : 1.f);
      float e[2][4];
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        const dq nj = snrm[s + l];
        const double dnx = nrm[0] - nj.x, dny = nrm[1] - nj.y, dnz = nrm[2] - nj.z;
        e[l][0] = (float)(-0.5 * dnx);
        e[l][1] = (float)(-0.5 * dny);
        e[l][2] = (float)(-0.5 * dnz);
        e[l][3] = (float)((nj.w - pin) + (cc[0] * dnx + cc[1] * dny + cc[2] * dnz));
      }
      EX = make_float2(e[0][0], e[1][0]);
      EY = make_float2(e[0][1], e[1][1]);
      EZ = make_float2(e[0][2], e[1][2]);
      EW = make_float2(e[0][3], e[1][3]);
    }
    const float4* r = srec + (size_t)(s >> 1) * kQ * kNrec * 2;
    float2 tj = sp_comp(r, 1, 2);  // J_j t_j of both triangles
    if constexpr (!FAR) tj = __fmul2_rn(tj, keep);
    float2 acc2[kQ], R[kQ];
#pragma unroll
    for (int a = 0; a < kQ; ++a) {
      acc2[a] = make_float2(0.f, 0.f);
      R[a] = make_float2(0.f, 0.f);
    }
    float2 Q2 = make_float2(0.f, 0.f);
#pragma unroll(kUnrollB)
    for (int b = 0; b < kQ; ++b) {
      const float4* rv = r + b * kNrec * 2;
      const float2 px = sp_comp(rv, 0, 0), py = sp_comp(rv, 0, 1), pz = sp_comp(rv, 0, 2), pw = sp_comp(rv, 0, 3);
      float2 sd = sp_comp(rv, 1, 0);
      if constexpr (!FAR) sd = __fmul2_rn(sd, keep);
      const float2 wb = bcast(wq[b]);
      float2 td = make_float2(0.f, 0.f);
#pragma unroll
      for (int a = 0; a < kQ; ++a) {
        float2 r2;
        if constexpr (FAR) {
          r2 = __ffma2_rn(X[a], px, __ffma2_rn(Y[a], py, __ffma2_rn(Z[a], pz, __fadd2_rn(W[a], pw))));
        } else {
          const float2 dx = __ffma2_rn(half2, px, X[a]);
          const float2 dy = __ffma2_rn(half2, py, Y[a]);
          const float2 dz = __ffma2_rn(half2, pz, Z[a]);
          r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, eps2)));
        }
        const float2 inv = make_float2(rsq(r2.x), rsq(r2.y));
        const float2 inv3 = __fmul2_rn(__fmul2_rn(inv, inv), inv);
        R[a] = __ffma2_rn(wb, inv, R[a]);
        acc2[a] = __ffma2_rn(sd, inv3, acc2[a]);
        td.x = fmaf(cd[a], inv3.x, td.x);
        td.y = fmaf(cd[a], inv3.y, td.y);
      }
      // e_i(y_b) for both lanes; y_b - c = -(1/2)(-2 y_b)
      const float2 e = __ffma2_rn(px, EX, __ffma2_rn(py, EY, __ffma2_rn(pz, EZ, EW)));
      Q2 = __ffma2_rn(__fmul2_rn(wb, e), td, Q2);
    }
    // single layer of both rows from R_a
    float2 U = make_float2(0.f, 0.f), S2 = make_float2(0.f, 0.f);
#pragma unroll
    for (int a = 0; a < kQ; ++a) {
      U = __ffma2_rn(bcast(wq[a]), R[a], U);
      S2 = __ffma2_rn(bcast(ca[a]), R[a], S2);
    }
    SLW = __ffma2_rn(tj, U, SLW);
    if constexpr (!FAR) {
      S2 = __fmul2_rn(S2, keep);
      Q2 = __fmul2_rn(Q2, keep);
    }
    red[s >> 1] = make_float4(S2.x, S2.y, Q2.x, Q2.y);
    // forward double layer: d_j(x_a) times the pair's sums (as eval_cell_sp)
    float2 nx, ny, nz, nw;
    if constexpr (FAR) {
      const float4 p0 = splane[s], p1 = splane[s + 1];
      nx = make_float2(p0.x, p1.x);
      ny = make_float2(p0.y, p1.y);
      nz = make_float2(p0.z, p1.z);
      nw = make_float2(-p0.w, -p1.w);
    } else {
      float pn[2][4];
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        const dq nj = snrm[s + l];
        const float dnx = (float)(nj.x - nrm[0]), dny = (float)(nj.y - nrm[1]), dnz = (float)(nj.z - nrm[2]);
        pn[l][0] = dnx;
        pn[l][1] = dny;
        pn[l][2] = dnz;
        pn[l][3] = (float)(cen[0] * nj.x + cen[1] * nj.y + cen[2] * nj.z - nj.w) + (o[0] * dnx + (o[1] * dny + o[2] * dnz));
      }
      nx = make_float2(pn[0][0], pn[1][0]);
      ny = make_float2(pn[0][1], pn[1][1]);
      nz = make_float2(pn[0][2], pn[1][2]);
      nw = make_float2(pn[0][3], pn[1][3]);
    }
#pragma unroll
    for (int a = 0; a < kQ; ++a) {
      const float2 d = __ffma2_rn(X[a], nx, __ffma2_rn(Y[a], ny, __ffma2_rn(Z[a], nz, nw)));
      DLp[a] = __ffma2_rn(d, acc2[a], DLp[a]);
    }
  }
  slw += SLW.x + SLW.y;
#pragma unroll
  for (int a = 0; a < kQ; ++a) dl[a] += DLp[a].x + DLp[a].y;
}

// FP64 form of eval_cell_sym (one source triangle at a time, the arithmetic
// of the FP64 ordered-pair kernel's eval_cell, the single layer through
// R_a): the transposed sums of triangle s go to red[s - s0] as (SL, DL).
template <bool FAR>
__device__ __forceinline__ void eval_cell_sym64(const dq* __restrict__ srec, const int4* __restrict__ svid,
                                                const dq* __restrict__ snrm, const dq* __restrict__ splane, int s0,
                                                int s1, int4 tv, const double (&x)[kQ], const double (&y)[kQ],
                                                const double (&z)[kQ], const double (&q2)[kQ],
                                                const double (&ca)[kQ], const double (&cd)[kQ],
                                                const double (&wq)[kQ], const double (&o)[3], const double (&cen)[3],
                                                const double (&nrm)[3], const double (&cc)[3], double pin,
                                                double& slw, double (&dl)[kQ], double2* __restrict__ red)
{
  double ex = 0.0, ey = 0.0, ez = 0.0, ew = 0.0;
  if constexpr (FAR) {
    ex = -0.5 * nrm[0];
    ey = -0.5 * nrm[1];
    ez = -0.5 * nrm[2];
    ew = cc[0] * nrm[0] + cc[1] * nrm[1] + cc[2] * nrm[2] - pin;
  }
#pragma unroll 1
  for (int s = s0; s < s1; ++s) {
    dq nj;
    if constexpr (!FAR) {
      if (shares_vertex(tv, svid[s])) {
        red[s - s0] = make_double2(0.0, 0.0);
        continue;
      }
      nj = snrm[s];
      const double dnx = nrm[0] - nj.x, dny = nrm[1] - nj.y, dnz = nrm[2] - nj.z;
      ex = -0.5 * dnx;
      ey = -0.5 * dny;
      ez = -0.5 * dnz;
      ew = (nj.w - pin) + (cc[0] * dnx + cc[1] * dny + cc[2] * dnz);
    }
    const dq* r = srec + (size_t)s * kQ * kNrec;
    const double tj = r[1].z;  // J_j t_j
    double acc[kQ], R[kQ];
#pragma unroll
    for (int a = 0; a < kQ; ++a) {
      acc[a] = 0.0;
      R[a] = 0.0;
    }
    double Qt = 0.0;
#pragma unroll(kUnrollB64)
    for (int b = 0; b < kQ; ++b) {
      const dq p0 = r[b * kNrec];
      const dq p1 = r[b * kNrec + 1];  // (s_b, c_b, J_j t_j, 0)
      double td = 0.0;
#pragma unroll
      for (int a = 0; a < kQ; ++a) {
        double r2;
        if constexpr (FAR) {
          r2 = x[a] * p0.x + (y[a] * p0.y + (z[a] * p0.z + (q2[a] + p0.w)));
        } else {
          const double dx = x[a] + 0.5 * p0.x, dy = y[a] + 0.5 * p0.y, dz = z[a] + 0.5 * p0.z;
          r2 = dx * dx + dy * dy + dz * dz;
        }
        const double inv = rsq_f64(r2);
        const double inv3 = (inv * inv) * inv;
        R[a] += wq[b] * inv;
        acc[a] += p1.x * inv3;
        td += cd[a] * inv3;
      }
      const double e = p0.x * ex + (p0.y * ey + (p0.z * ez + ew));
      Qt += (wq[b] * e) * td;
    }
    double U = 0.0, S = 0.0;
#pragma unroll
    for (int a = 0; a < kQ; ++a) {
      U += wq[a] * R[a];
      S += ca[a] * R[a];
    }
    slw += tj * U;
    red[s - s0] = make_double2(S, Qt);
    // forward double layer (as eval_cell)
    if constexpr (FAR) {
      const dq pn = splane[s];
#pragma unroll
      for (int a = 0; a < kQ; ++a) dl[a] += (x[a] * pn.x + (y[a] * pn.y + (z[a] * pn.z - pn.w))) * acc[a];
    } else {
      const double dnx = nj.x - nrm[0], dny = nj.y - nrm[1], dnz = nj.z - nrm[2];
      const double e0 = (cen[0] * nj.x + cen[1] * nj.y + cen[2] * nj.z - nj.w) + (o[0] * dnx + (o[1] * dny + o[2] * dnz));
#pragma unroll
      for (int a = 0; a < kQ; ++a) dl[a] += (x[a] * dnx + (y[a] * dny + (z[a] * dnz + e0))) * acc[a];
    }
  }
}

// Single layer only with NC right-hand sides (FP32): one sum R_a per pair and
// target point whatever NC; the columns differ in the per-pair folds.
template <int NC, bool FAR>
__device__ __forceinline__ void eval_cell_sym_sl(const float4* __restrict__ srec, const int4* __restrict__ svid,
                                                 int s0, int s1, int4 tv, const float (&x)[kQ],
                                                 const float (&y)[kQ], const float (&z)[kQ],
                                                 const float (&q2)[kQ], const float (&cw)[NC][kQ],
                                                 const float (&om)[kQ], const float (&wq)[kQ], float (&slw)[NC],
                                                 float2* __restrict__ red)
{
  float2 X[kQ], Y[kQ], Z[kQ], W[kQ];
#pragma unroll
  for (int a = 0; a < kQ; ++a) {
    X[a] = bcast(x[a]);
    Y[a] = bcast(y[a]);
    Z[a] = bcast(z[a]);
    W[a] = bcast(q2[a]);
  }
  float2 SLW[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) SLW[c] = make_float2(0.f, 0.f);
  const float2 half2 = bcast(0.5f);
  const float2 eps2 = bcast(1e-24f);
#pragma unroll 1
  for (int s = s0; s < s1; s += 2) {
    float2 keep = make_float2(1.f, 1.f);
    if constexpr (!FAR) {
      const bool m0 = shares_vertex(tv, svid[s]), m1 = shares_vertex(tv, svid[s + 1]);
      if (m0 && m1) {
#pragma unroll
        for (int c = 0; c < NC; ++c) red[(s >> 1) * NC + c] = make_float2(0.f, 0.f);
        continue;
      }
      keep = make_float2(m0 ? 0.f : 1.f, m1 ? 0.f : 1.f);
    }
    const float4* r = srec + (size_t)(s >> 1) * kQ * kNrec * 2;
    float2 R[kQ];
#pragma unroll
    for (int a = 0; a < kQ; ++a) R[a] = make_float2(0.f, 0.f);
#pragma unroll
    for (int b = 0; b < kQ; ++b) {
      const float4* rv = r + b * kNrec * 2;
      const float2 px = sp_comp(rv, 0, 0), py = sp_comp(rv, 0, 1), pz = sp_comp(rv, 0, 2), pw = sp_comp(rv, 0, 3);
      const float2 ob = bcast(om[b]);
#pragma unroll
      for (int a = 0; a < kQ; ++a) {
        float2 r2;
        if constexpr (FAR) {
          r2 = __ffma2_rn(X[a], px, __ffma2_rn(Y[a], py, __ffma2_rn(Z[a], pz, __fadd2_rn(W[a], pw))));
        } else {
          const float2 dx = __ffma2_rn(half2, px, X[a]);
          const float2 dy = __ffma2_rn(half2, py, Y[a]);
          const float2 dz = __ffma2_rn(half2, pz, Z[a]);
          r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, eps2)));
        }
        const float2 inv = make_float2(rsq(r2.x), rsq(r2.y));
        R[a] = __ffma2_rn(ob, inv, R[a]);
      }
    }
    float2 U = make_float2(0.f, 0.f);
#pragma unroll
    for (int a = 0; a < kQ; ++a) U = __ffma2_rn(bcast(wq[a]), R[a], U);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      float2 c0 = sp_comp(r, 1, c);  // first-point charges of both triangles
      if constexpr (!FAR) c0 = __fmul2_rn(c0, keep);
      SLW[c] = __ffma2_rn(c0, U, SLW[c]);
      float2 S = make_float2(0.f, 0.f);
#pragma unroll
      for (int a = 0; a < kQ; ++a) {
        S.x = fmaf(cw[c][a], R[a].x, S.x);
        S.y = fmaf(cw[c][a], R[a].y, S.y);
      }
      if constexpr (!FAR) S = __fmul2_rn(S, keep);
      red[(s >> 1) * NC + c] = S;
    }
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) slw[c] += SLW[c].x + SLW[c].y;
}

// The same in FP64, one source triangle at a time.
template <int NC, bool FAR>
__device__ __forceinline__ void eval_cell_sym64_sl(const dq* __restrict__ srec, const int4* __restrict__ svid, int s0,
                                                   int s1, int4 tv, const double (&x)[kQ], const double (&y)[kQ],
                                                   const double (&z)[kQ], const double (&q2)[kQ],
                                                   const double (&cw)[NC][kQ], const double (&om)[kQ],
                                                   const double (&wq)[kQ], double (&slw)[NC],
                                                   double* __restrict__ red)
{
#pragma unroll 1
  for (int s = s0; s < s1; ++s) {
    if constexpr (!FAR) {
      if (shares_vertex(tv, svid[s])) {
#pragma unroll
        for (int c = 0; c < NC; ++c) red[(s - s0) * NC + c] = 0.0;
        continue;
      }
    }
    const dq* r = srec + (size_t)s * kQ * kNrec;
    double R[kQ];
#pragma unroll
    for (int a = 0; a < kQ; ++a) R[a] = 0.0;
#pragma unroll(kUnrollB64)
    for (int b = 0; b < kQ; ++b) {
      const dq p0 = r[b * kNrec];
#pragma unroll
      for (int a = 0; a < kQ; ++a) {
        double r2;
        if constexpr (FAR) {
          r2 = x[a] * p0.x + (y[a] * p0.y + (z[a] * p0.z + (q2[a] + p0.w)));
        } else {
          const double dx = x[a] + 0.5 * p0.x, dy = y[a] + 0.5 * p0.y, dz = z[a] + 0.5 * p0.z;
          r2 = dx * dx + dy * dy + dz * dz;
        }
        R[a] += om[b] * rsq_f64(r2);
      }
    }
    double U = 0.0;
#pragma unroll
    for (int a = 0; a < kQ; ++a) U += wq[a] * R[a];
    const dq p1 = r[1];  // first-point charges
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      slw[c] += comp(p1, c) * U;
      double S = 0.0;
#pragma unroll
      for (int a = 0; a < kQ; ++a) S += cw[c][a] * R[a];
      red[(s - s0) * NC + c] = S;
    }
  }
}

}  // namespace eb
