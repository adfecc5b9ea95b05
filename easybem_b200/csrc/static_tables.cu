// Static tables of a mesh on the GPU, from its vertices, triangles, sorted
// order and cell balls.
//
// Built on the host and copied (1.3 KB a triangle through pinned staging) they
// took 2.3 ms of a new 5,000-triangle mesh; the inputs are 80 bytes a triangle
// and one thread per triangle writes its rows, bound by the stores.
#include <cuda_runtime.h>

#include "engine.h"

namespace eb {

__global__ void __launch_bounds__(128) static_tables_kernel(StaticTables t)
{
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  double rho2 = 0.0;
  if (s < t.ne) {
    const int orig = t.perm[s];
    const int f[3] = {t.elems[3 * (size_t)orig], t.elems[3 * (size_t)orig + 1], t.elems[3 * (size_t)orig + 2]};
    d3 P[3];
    for (int k = 0; k < 3; k++)
      P[k] = mk3(t.nodes[3 * (size_t)f[k]], t.nodes[3 * (size_t)f[k] + 1], t.nodes[3 * (size_t)f[k] + 2]);
    const d3 w = P[1] - P[0], z = P[2] - P[0];
    const d3 n = cross3(w, z);
    const double J = sqrt(dot3(n, n));
    const d3 nu = mk3(n.x / J, n.y / J, n.z / J);
    t.trin[s] = dq{nu.x, nu.y, nu.z, J};
    t.snrm[s] = dq{nu.x, nu.y, nu.z, dot3(P[0], nu)};
    const int4 vid = make_int4(f[0], f[1], f[2], 0);
    t.svid[s] = vid;
    const dq cb = t.ccent[s / kCell];
    const d3 cc = mk3(cb.x, cb.y, cb.z);
    const double hp = dot3(P[0] - cc, nu);
    t.splane64[s] = dq{nu.x, nu.y, nu.z, hp};
    t.splane32[s] = make_float4((float)nu.x, (float)nu.y, (float)nu.z, (float)hp);
    for (int b = 0; b < t.Q; b++) {
      const d3 y = P[0] + t.bary[2 * b] * w + t.bary[2 * b + 1] * z;
      const size_t i = (size_t)s * t.Q + b;
      t.wj[i] = t.tw[b] * J;
      const d3 yr = y - cc;
      const double y2 = dot3(yr, yr);
      rho2 = fmax(rho2, y2);
      t.pos64[i] = dq{-2.0 * yr.x, -2.0 * yr.y, -2.0 * yr.z, y2};
      const float fx = (float)yr.x, fy = (float)yr.y, fz = (float)yr.z;
      t.pos32[i] = make_float4(-2.0f * fx, -2.0f * fy, -2.0f * fz,
                               (float)((double)fx * fx + (double)fy * fy + (double)fz * fz));
    }
    const d3 cen = (1.0 / 3.0) * (P[0] + P[1] + P[2]);
    for (int ch = 0; ch < t.nchunk; ch++) {
      const size_t item = (size_t)s * t.nchunk + ch;
      t.tcent[item] = dq{cen.x, cen.y, cen.z, 0.0};
      t.tnrm[item] = dq{nu.x, nu.y, nu.z, 0.0};
      t.tvid[item] = vid;
      for (int a = 0; a < t.K; a++) {
        const int pa = ch * t.K + a, pp = min(pa, t.Q - 1);
        const double wa = pa < t.Q ? t.tw[pp] : 0.0, e1 = t.bary[2 * pp], e2 = t.bary[2 * pp + 1];
        const d3 xr = P[0] + e1 * w + e2 * z - cen;
        const size_t i = item * t.K + a;
        t.tgt64[i] = dq{xr.x, xr.y, xr.z, wa};
        t.tgt32[i] = make_float4((float)xr.x, (float)xr.y, (float)xr.z, (float)wa);
        // P1 test weights w_a (1 - xi - eta, xi, eta) in the triangle's vertex order
        const double p0 = wa * (1.0 - e1 - e2), p1 = wa * e1, p2 = wa * e2;
        t.tgtw64[i] = dq{p0, p1, p2, 0.0};
        t.tgtw32[i] = make_float4((float)p0, (float)p1, (float)p2, 0.0f);
      }
    }
  }
  // a warp is a cell: its radius over the quadrature points
  for (int o = 16; o; o >>= 1) rho2 = fmax(rho2, __shfl_xor_sync(0xffffffffu, rho2, o));
  if ((threadIdx.x & 31) == 0 && s < t.ne) t.rho[s / kCell] = sqrt(rho2) * (1.0 + 1e-12);
}

// Balls around the triangles of n consecutive target items (one warp each):
// the box centre, moved towards the farthest vertex four times (vertex_ball).
__global__ void item_balls_kernel(StaticTables t, int n, int count, dq* __restrict__ out)
{
  const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (g >= count) return;
  const int i0 = g * n, i1 = min(t.ne * t.nchunk, i0 + n);
  const int v0 = 3 * (i0 / t.nchunk), v1 = 3 * ((i1 - 1) / t.nchunk + 1);
  auto vertex = [&](int v) {
    const int k = t.elems[3 * (size_t)t.perm[v / 3] + v % 3];
    return mk3(t.nodes[3 * (size_t)k], t.nodes[3 * (size_t)k + 1], t.nodes[3 * (size_t)k + 2]);
  };
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  for (int v = v0 + lane; v < v1; v += 32) {
    const d3 p = vertex(v);
    const double c[3] = {p.x, p.y, p.z};
    for (int d = 0; d < 3; d++) {
      lo[d] = fmin(lo[d], c[d]);
      hi[d] = fmax(hi[d], c[d]);
    }
  }
  for (int d = 0; d < 3; d++)
    for (int o = 16; o; o >>= 1) {
      lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
      hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
    }
  d3 c = mk3(0.5 * (lo[0] + hi[0]), 0.5 * (lo[1] + hi[1]), 0.5 * (lo[2] + hi[2])), best = c;
  double best2 = -1.0;
  for (int it = 0; it <= 4; it++) {
    double r2 = -1.0;
    int far = v1;
    for (int v = v0 + lane; v < v1; v += 32) {
      const d3 e = vertex(v) - c;
      const double d2 = dot3(e, e);
      if (d2 > r2) {
        r2 = d2;
        far = v;
      }
    }
    for (int o = 16; o; o >>= 1) {
      const double x = __shfl_xor_sync(0xffffffffu, r2, o);
      const int y = __shfl_xor_sync(0xffffffffu, far, o);
      if (x > r2 || (x == r2 && y < far)) {
        r2 = x;
        far = y;
      }
    }
    if (best2 < 0.0 || r2 < best2) {
      best2 = r2;
      best = c;
    }
    c = c + (1.0 / (it + 4.0)) * (vertex(far) - c);
  }
  if (lane == 0) out[g] = dq{best.x, best.y, best.z, sqrt(best2) * (1.0 + 1e-12)};
}

cudaError_t static_tables_launch(const StaticTables& t, cudaStream_t st)
{
  static_tables_kernel<<<(t.ne + 127) / 128, 128, 0, st>>>(t);
  const int items = t.ne * t.nchunk;
  const int tiles = (items + kTT - 1) / kTT, warps = (items + kWarpItems - 1) / kWarpItems;
  item_balls_kernel<<<(tiles + 3) / 4, 128, 0, st>>>(t, kTT, tiles, t.ttile);
  static_assert(kWarpItems == kCell, "a warp of one-item triangles is a cell");
  if (t.nchunk > 1) item_balls_kernel<<<(warps + 3) / 4, 128, 0, st>>>(t, kWarpItems, warps, t.twarp);
  else cudaMemcpyAsync(t.twarp, t.ccent, sizeof(dq) * warps, cudaMemcpyDeviceToDevice, st);
  return cudaGetLastError();
}

}  // namespace eb
