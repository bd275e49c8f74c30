// Householder reduction of a mid-sized matrix (up to 64 x 64 tiles in number of what two CTAs per SM hold, n = 1472 on
// 148 SMs) in one cooperative launch, the matrix held in registers: the per-CTA reduction of cta_eigen.cuh spread over
// the GPU. CTA c owns one tile (I, J), I >= J, of the lower triangle (a diagonal tile holds both triangles), thread
// (ty, tx) of its 16 x 16 grid the elements (ty + 16 a, tx + 16 b). Tiles are numbered from the last
// corner, so the tiles that still meet the trailing block are always the first ones; the others leave.
//
// The reflector of column i is H = I - tau v v^T with v = x - beta e_{i+1}, x the column below the diagonal, so the products A x
// need no scalars. Per column two grid-wide barriers:
//   1  every tile: row and column sums of A x into its slot, its part of x^T A x, the present values of column i + 1.
//   2  the diagonal tiles, as owners of their 64 rows: y from the slots, w = tau y + a2 v, and the updated next
//      column with its norm part (A_{i+1} - v w_{i+1} - w v_{i+1}).
//   then every tile reads v, w and the next column for its rows and columns, updates its registers and goes on.
// What bounds it: the barriers and the L2 round trips behind them, 4.7 us a column at n = 966; the panel kernel
// (panel_coop.cuh), which streams the trailing block from L2 for every column, takes 13.2 us.
// Data written by another CTA is read through L2 (ld.global.cg). Every sum runs in a fixed order.
#pragma once
#include "panel_coop.cuh"

namespace pm3gpu {
namespace large {

constexpr int kTileParts = 10;  // column partials by warp: 16-byte rows without bank conflicts

// Barrier of the first `act` CTAs: a counter that only grows; `target` is its value once all have arrived. Bounded: after about
// 2^22 polls (a second or two) the wait raises gs->err, and every CTA that waits leaves the same way.
__device__ __forceinline__ bool tile_sync(GridSync* gs, unsigned int target) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.add.release.gpu.u32 [%0], 1;" ::"l"(&gs->count) : "memory");
    bool ok = false;
    for (unsigned int spin = 0; spin < (1u << 22); ++spin) {
      if ((int)(ld_acquire_u32(&gs->count) - target) >= 0) {
        ok = true;
        break;
      }
    }
    if (!ok) atomicExch(&gs->err, 1);
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

constexpr int kTileMaxStripes = 23;  // step 2 loads the slots of a row 6 x 4 at a time, the parts of x^T A x 9 x 32
__host__ __device__ constexpr int tile_stripes(int n) { return (n + kTile - 1) / kTile; }
// doubles of exchange buffer beside the tile slots: the column (two generations), w, the next column's old values,
// norm parts, parts of x^T A x, v_{i+1}
__host__ __device__ constexpr size_t tile_exchange(int n) {
  const size_t t = (size_t)tile_stripes(n);
  return 4 * t * kTile + 2 * t + t * (t + 1) / 2 + 8;
}

__global__ void __launch_bounds__(kBlock, 2)
    tile_reduce_kernel(double* __restrict__ A, int n, double* __restrict__ d, double* __restrict__ e, double* __restrict__ tau,
                       double* tp, double* buf, GridSync* gs) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tx = tid & 15, ty = tid >> 4;
  const int nts = tile_stripes(n), M = nts * kTile, c = blockIdx.x;
  int Jr = (int)((sqrtf(8.0f * c + 1.0f) - 1.0f) * 0.5f);
  while (Jr * (Jr + 1) / 2 > c) --Jr;
  while ((Jr + 1) * (Jr + 2) / 2 <= c) ++Jr;
  const int J = nts - 1 - Jr, I = nts - 1 - (c - Jr * (Jr + 1) / 2);
  const bool diag = I == J;
  double* xs = buf;               // [2][M]
  double* ws = xs + 2 * M;        // [M]
  double* raw = ws + M;           // [M]
  double* npart = raw + M;        // [2 nts]
  double* qp = npart + 2 * nts;   // [tiles]
  double* v1g = qp + nts * (nts + 1) / 2;
  auto slot = [&](int i2, int j2) { return tp + ((size_t)i2 * (i2 + 1) / 2 + j2) * (2 * kTile); };
  __shared__ double xb[2][2 * kTile];  // the column over the tile's rows, then its columns (two generations)
  __shared__ double wb[2 * kTile];
  __shared__ __align__(16) double cpart[kTile * kTileParts];
  __shared__ __align__(16) double qs[8];
  __shared__ double zg[4][kTile];
  __shared__ double sc[8];  // beta, tau, v1; z_{i+1}, x^T A x, raw_{i+1}
  double a[4][4];
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = I * kTile + ty + 16 * p, col = J * kTile + tx + 16 * q, hi = max(r, col), lo = min(r, col);
      a[p][q] = hi < n ? A[(size_t)hi * n + lo] : 0.0;
    }
  unsigned int target = gridDim.x;
  if (J == 0 && tx == 0) {
#pragma unroll
    for (int p = 0; p < 4; ++p) raw[I * kTile + ty + 16 * p] = a[p][0];
  }
  if (!tile_sync(gs, target)) return;
  if (diag && tid < kTile) {
    const int p = I * kTile + tid;
    const double r0 = __ldcg(raw + p), x = p > 0 ? r0 : 0.0;
    xs[p] = x;
    if (p == 0) d[0] = r0;
    const double part = warp_sum(p > 1 ? x * x : 0.0);
    if (lane == 0) npart[2 * I + warp] = part;
  }
  target += gridDim.x;
  if (!tile_sync(gs, target)) return;
  if (tid < 2 * kTile) xb[0][tid] = __ldcg(xs + (tid < kTile ? I : J) * kTile + (tid & (kTile - 1)));
  __syncthreads();
  int par = 0;
  for (int i = 0; i < n - 2; ++i) {
    const int I0 = (i + 1) / kTile, ntr = nts - I0, act = ntr * (ntr + 1) / 2;
    if (c >= act) return;
    // ------------------------------------------------------------------ 1: products
    if (diag && warp == 7) {  // the reflector's scalars, for step 2
      double x0 = lane < 2 * ntr ? __ldcg(npart + 2 * I0 + lane) : 0.0;
      if (lane + 32 < 2 * ntr) x0 += __ldcg(npart + 2 * I0 + lane + 32);
      const double alpha = __ldcg(xs + (size_t)par * M + i + 1), xn2 = warp_sum(x0);
      if (lane == 0) {
        const bool zero = !(xn2 > 1.0e-240);
        const double s = fma(alpha, alpha, xn2), nrm = sqrt(s);
        const double beta = zero ? alpha : -copysign(nrm, alpha);
        sc[0] = beta;
        sc[1] = zero ? 0.0 : 1.0 / fma(fabs(alpha), nrm, s);
        sc[2] = alpha - beta;
      }
    }
    {
      const double* xI = xb[par];
      const double* xJ = xI + kTile;
      double vc[4], pc[4], py[8], dot = 0.0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        vc[q] = xJ[tx + 16 * q];
        pc[q] = 0.0;
      }
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const double vr = xI[ty + 16 * p];
        double acc = 0.0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          acc = fma(a[p][q], vc[q], acc);
          pc[q] = fma(a[p][q], vr, pc[q]);
        }
        dot = fma(acc, vr, dot);
        py[p] = acc;
      }
      if (!diag) dot *= 2.0;  // the tile stands for both triangles
      py[4] = dot;
      py[5] = py[6] = py[7] = 0.0;
      if (J == I0 && tx == ((i + 1) & 15)) {
        const int q = ((i + 1) & (kTile - 1)) >> 4;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const double r = q == 0 ? a[p][0] : (q == 1 ? a[p][1] : (q == 2 ? a[p][2] : a[p][3]));
          raw[I * kTile + ty + 16 * p] = r;
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) pc[q] += __shfl_xor_sync(0xffffffffu, pc[q], 16);
      if (!diag && lane < 16) {
#pragma unroll
        for (int q = 0; q < 4; ++q) cpart[(tx + 16 * q) * kTileParts + warp] = pc[q];
      }
      const double sum = sum16_of8(py, lane);
      const double both = sum + __shfl_xor_sync(0xffffffffu, sum, 16);
      const int k = (lane & 15) >> 1;
      if (!(lane & 1)) {
        if (k < 4) slot(I, J)[ty + 16 * k] = sum;
        else if (k == 4 && lane < 16) qs[warp] = both;
      }
    }
    __syncthreads();
    if (!diag && tid < kTile) slot(I, J)[kTile + tid] = sum8(cpart + tid * kTileParts);
    if (tid == kTile) qp[c] = sum8(qs);
    target += act;
    if (!tile_sync(gs, target)) return;
    // ------------------------------------------------------------------ 2: the owners' rows
    if (diag) {
      const int g = tid >> 6, r = tid & (kTile - 1), p = I * kTile + r;
      double z[6];
#pragma unroll
      for (int u = 0; u < 6; ++u) {
        const int t = I0 + g + 4 * u;
        z[u] = t < nts ? __ldcg(t <= I ? slot(I, t) + r : slot(t, I) + kTile + r) : 0.0;
      }
      const double raw0 = g == 0 ? __ldcg(raw + p) : 0.0;
      if (warp == 7) {  // row i + 1 of A x
        const int t = I0 + lane, o = (i + 1) & (kTile - 1);
        const double v = warp_sum(t < nts ? __ldcg(t == I0 ? slot(I0, I0) + o : slot(t, I0) + kTile + o) : 0.0);
        if (lane == 0) sc[3] = v;
      } else if (warp == 6) {
        double v[9];
#pragma unroll
        for (int u = 0; u < 9; ++u) v[u] = lane + 32 * u < act ? __ldcg(qp + lane + 32 * u) : 0.0;
        const double t = warp_sum(((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7])) + v[8]);
        if (lane == 0) sc[4] = t;
      } else if (tid == 160) {
        sc[5] = __ldcg(raw + i + 1);
      }
      zg[g][r] = ((z[0] + z[1]) + (z[2] + z[3])) + (z[4] + z[5]);
      __syncthreads();
      if (tid < kTile) {
        const double beta = sc[0], tt = sc[1], v1 = sc[2], z1 = sc[3], q = sc[4], raw1 = sc[5];
        const double zz = (zg[0][r] + zg[1][r]) + (zg[2][r] + zg[3][r]);
        const double y1 = fma(-beta, raw1, z1), y = fma(-beta, raw0, zz);
        const double vav = fma(-beta, z1 + y1, q);
        const double a2 = -0.5 * tt * tt * vav;
        const double v = p == i + 1 ? v1 : xb[par][r];
        const double w = p > i ? fma(tt, y, a2 * v) : 0.0;
        const double w1 = fma(tt, y1, a2 * v1);
        const double x = raw0 - fma(v, w1, w * v1);
        xs[(size_t)(1 - par) * M + p] = p > i + 1 ? x : 0.0;
        ws[p] = w;
        const double part = warp_sum(p > i + 2 ? x * x : 0.0);
        if (lane == 0) npart[2 * I + warp] = part;
        if (p == i + 1) {
          *v1g = v1;
          d[i + 1] = x;
          e[i] = beta;
          tau[i] = tt * v1 * v1;  // of the reflector scaled to v_{i+1} = 1, as the back-transformation takes it
        }
      }
    }
    target += act;
    if (!tile_sync(gs, target)) return;
    // ------------------------------------------------------------------ update, next column
    {
      const int k = tid & (2 * kTile - 1), at = (k < kTile ? I : J) * kTile + (k & (kTile - 1));
      const double v1 = __ldcg(v1g);
      const double in = tid < 2 * kTile ? __ldcg(ws + at) : __ldcg(xs + (size_t)(1 - par) * M + at);
      if (diag && tid < kTile) {  // the stored reflector
        const int p = I * kTile + tid;
        if (p > i + 1 && p < n) A[(size_t)i * n + p] = sc[1] != 0.0 ? xb[par][tid] / v1 : 0.0;
      }
      if (tid < 2 * kTile) wb[k] = in;
      else xb[1 - par][k] = in;
      __syncthreads();
      const double* xI = xb[par];
      const double* xJ = xI + kTile;
      double vr[4], wr[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        vr[p] = I * kTile + ty + 16 * p == i + 1 ? v1 : xI[ty + 16 * p];
        wr[p] = wb[ty + 16 * p];
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double vcq = J * kTile + tx + 16 * q == i + 1 ? v1 : xJ[tx + 16 * q], wcq = wb[kTile + tx + 16 * q];
#pragma unroll
        for (int p = 0; p < 4; ++p) a[p][q] = fma(-wr[p], vcq, fma(-vr[p], wcq, a[p][q]));
      }
    }
    par = 1 - par;
  }
  if (c == 0) {  // the last corner
    const int r = n - 1 - I * kTile;
    if (tid == 0) {
      e[n - 2] = __ldcg(xs + (size_t)par * M + n - 1);
      tau[n - 2] = 0.0;
      e[n - 1] = 0.0;
    }
    if (ty == (r & 15) && tx == (r & 15)) {
      const int q = r >> 4;
      d[n - 1] = q == 0 ? a[0][0] : (q == 1 ? a[1][1] : (q == 2 ? a[2][2] : a[3][3]));
    }
  }
}

}  // namespace large
}  // namespace pm3gpu
