// The numerics of a solve under the reference's second-derivative tolerances (pm3-rs src/hessian.rs:169-175: e_tol <= 1e-12,
// p_tol <= 1e-11, max_scf >= 500): what scf_tight_kernel runs in place of scf_kernel.cuh's and cta_eigen.cuh's.
//
// Such a solve is one end of a difference over 2e-3 Bohr, which turns 1e-11 of its density into 1e-9 of a Hessian. Near the end
// of the iteration the accelerator's error vectors are nearly parallel, and its pivot guard (1e-12 of the scaled Gram matrix)
// passes or fails by their rounding: where it passes the state lands within 1e-15, where it fails the iteration stops with
// up to 1e-11 left. So another order of the same sums is another Hessian. scf_kernel.cuh's sums moved those of an 8-atom organic
// by up to 1.8e-9 relative (24 geometries, 7 of them beyond 1e-9); those kept here, every product, reduction and division in its
// order and form, give them back to 2e-12. The dipole derivatives of the same molecule moved by up to 1.2e-6 and are equal
// again. Molecules of up to 32 atom pairs (one warp's) repeat to 1e-14; with more, the order of the atomic sums between warps
// varies, and two runs of an 11-atom molecule differ by up to 3e-9. The cost: 5.4 ms against 3.1 for three molecules of 8-14 atoms
// (198 solves).
//
// The eigensolver is the same chain as in cta_eigen.cuh (Householder, multisection, twisted vectors, back-transformation) on a
// packed lower triangle (row-major: element (r, c), r >= c, at r(r+1)/2 + c) in shared memory, or in global memory when it does not fit.
#pragma once
#include "scf_kernel.cuh"

namespace pm3gpu {
namespace tight {

// ------------------------------------------------------------------------- products
constexpr int kGemmScratch = 2 * 16 * 65;  // doubles of cta_gemm's tiles

// This thread's 4 + 4 elements of the 64 x 16 chunks of op(A) and op(B) at k0 (the layout of
// cta_gemm's shared tiles), zero outside the matrices.
template <bool TA>
__device__ __forceinline__ void cta_gemm_fetch(double (&pa)[4], double (&pb)[4], int k0, int i0, int j0, int m, int n,
                                               int k, const double* __restrict__ A, int lda,
                                               const double* __restrict__ B, int ldb) {
  constexpr int BM = 64, BN = 64, BK = 16;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int e = threadIdx.x + q * kThreads;
    int ii, kk;
    if (TA) { ii = e % BM; kk = e / BM; } else { kk = e % BK; ii = e / BK; }
    const int gi = i0 + ii, gk = k0 + kk;
    pa[q] = (gi < m && gk < k) ? (TA ? A[(size_t)gk * lda + gi] : A[(size_t)gi * lda + gk]) : 0.0;
    const int jj = e % BN;
    kk = e / BN;
    const int gj = j0 + jj, gk2 = k0 + kk;
    pb[q] = (gj < n && gk2 < k) ? B[(size_t)gk2 * ldb + gj] : 0.0;
  }
}

// C (m x n) = alpha * op(A) * op(B) with op(A) m x k, op(B) k x n; A, B row-major in global
// memory. TA: A stored as k x m (use its transpose). Each output element goes through
// `epi(i, j, value)`. Tiles of 64 x 64, k-chunks of 16 (the next chunk's loads in flight while the
// current one is multiplied), 4 x 4 outputs per thread; `tile` needs 2 * 64 * 17 doubles of shared
// memory. If `lower_only`, only tiles touching the lower
// triangle (i >= j) are computed (for symmetric results).
template <bool TA, class Epi>
__device__ void cta_gemm(int m, int n, int k, double alpha, const double* __restrict__ A, int lda,
                         const double* __restrict__ B, int ldb, double* tile, bool lower_only, Epi epi) {
  constexpr int BM = 64, BN = 64, BK = 16;
  double* As = tile;              // [BK][BM+1]
  double* Bs = tile + BK * (BM + 1);  // [BK][BN+1]
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;  // 16 x 16 threads
  const int tiles_m = (m + BM - 1) / BM, tiles_n = (n + BN - 1) / BN;
  for (int t = 0; t < tiles_m * tiles_n; ++t) {
    const int bi = t / tiles_n, bj = t % tiles_n;
    if (lower_only && bj > bi) continue;  // uniform across the CTA
    const int i0 = bi * BM, j0 = bj * BN;
    double acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;
    // the next k-chunk's elements are loaded into registers while the current one is multiplied
    // (each thread holds 4 of op(A) and 4 of op(B): 64 x 16 / 256 threads)
    double pa[4], pb[4];
    cta_gemm_fetch<TA>(pa, pb, 0, i0, j0, m, n, k, A, lda, B, ldb);
    for (int k0 = 0; k0 < k; k0 += BK) {
      __syncthreads();  // the previous chunk's products have read As, Bs
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int e = threadIdx.x + q * kThreads;
        int ii, kk;
        if (TA) { ii = e % BM; kk = e / BM; } else { kk = e % BK; ii = e / BK; }
        As[kk * (BM + 1) + ii] = pa[q];
        const int jj = e % BN;
        kk = e / BN;
        Bs[kk * (BN + 1) + jj] = pb[q];
      }
      __syncthreads();
      if (k0 + BK < k) cta_gemm_fetch<TA>(pa, pb, k0 + BK, i0, j0, m, n, k, A, lda, B, ldb);
#pragma unroll
      for (int kk = 0; kk < BK; ++kk) {
        double a[4], b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          a[q] = As[kk * (BM + 1) + ty + 16 * q];
          b[q] = Bs[kk * (BN + 1) + tx + 16 * q];
        }
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[p][q] = fma(a[p], b[q], acc[p][q]);
      }
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int gi = i0 + ty + 16 * p, gj = j0 + tx + 16 * q;
        if (gi < m && gj < n) epi(gi, gj, alpha * acc[p][q]);
      }
  }
  __syncthreads();
}

// ---------------------------------------------------------------------- eigensolver
constexpr int kRowT = kMaxN / 32;   // rows per lane of a warp

__device__ __forceinline__ int tri(int r) { return r * (r + 1) / 2; }

// Sum over the CTA with one barrier: `red` holds two alternating kWarps buffers, so a call may
// overwrite the buffer two calls back without waiting (the previous call's barrier separates them).
__device__ __forceinline__ double block_sum_alt(double v, double* red, int& parity) {
  v = warp_sum(v);
  double* buf = red + parity * kWarps;
  parity ^= 1;
  if ((threadIdx.x & 31) == 0) buf[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
#pragma unroll
  for (int i = 0; i < kWarps; ++i) t += buf[i];
  return t;
}

// Householder reduction (n <= kThreads). For column i, the m = n - i - 1 trailing rows get T
// threads each (T the largest power of two with T m <= kThreads, at most a warp), so that late
// columns, with few rows left, still keep the CTA busy. The T threads of row r split the
// matrix-vector product (its row segment c <= r, then the column below it) and the rank-2
// update of its row segment by interleaved columns, and combine the product by shuffles; the
// first of them contributes its element of the next column to the next reflector's norm.
// Three barriers per column. This sweep reduces columns [0, i_stop) of the n x n matrix and, with
// `close`, writes the last diagonal and off-diagonal entries; d, e, tau are indexed from the
// matrix's first row.
__device__ __forceinline__ void householder_columns(int n, double* __restrict__ A, double* v, double* p, double* red, double* tau_out,
                                    double* e_out, double* d_out, int i_stop, bool close) {
  // scratch pointers in registers: the stores below go through generic pointers, which
  // would otherwise force them to be re-read after every store
  struct {
    double *v, *p, *red, *tau, *e, *d;
  } s = {v, p, red, tau_out, e_out, d_out};
  const int t = threadIdx.x;
  int parity = 0;
  double xn2 = block_sum_alt(t >= 2 && t < n ? A[tri(t)] * A[tri(t)] : 0.0, s.red, parity);
  for (int i = 0; i < i_stop; ++i) {
    const double alpha = A[tri(i + 1) + i];
    double beta = alpha, tau = 0.0, scal = 0.0;
    if (xn2 > 0.0) {
      beta = -copysign(sqrt(alpha * alpha + xn2), alpha);
      tau = (beta - alpha) / beta;
      scal = 1.0 / (alpha - beta);
    }
    if (t == 0) {
      s.tau[i] = tau;
      s.e[i] = beta;
      s.d[i] = A[tri(i) + i];
    }
    if (xn2 == 0.0) {  // column already reduced (uniform): only the next norm is needed
      xn2 = block_sum_alt(t >= i + 3 && t < n ? A[tri(t) + i + 1] * A[tri(t) + i + 1] : 0.0, s.red, parity);
      continue;
    }
    if (t > i && t < n) {  // reflector: one thread per row
      double vr = 1.0;
      if (t > i + 1) {
        vr = A[tri(t) + i] * scal;
        A[tri(t) + i] = vr;
      }
      s.v[t] = vr;
    }
    __syncthreads();
    const int m = n - i - 1;
    const int lg = min(5, 31 - __clz(kThreads / m));
    const int T = 1 << lg, k = t & (T - 1), r = i + 1 + (t >> lg);
    const bool mine = r < n;
    const int tr = mine ? tri(r) : 0;
    // y_r = sum_{c > i} A(r, c) v_c; four independent accumulators per thread
    double y = 0.0;
    if (mine) {
      double y0 = 0.0, y1 = 0.0, y2 = 0.0, y3 = 0.0;
      const double* row = A + tr;
      int c = i + 1 + k;
      for (; c + 3 * T <= r; c += 4 * T) {
        y0 = fma(row[c], s.v[c], y0);
        y1 = fma(row[c + T], s.v[c + T], y1);
        y2 = fma(row[c + 2 * T], s.v[c + 2 * T], y2);
        y3 = fma(row[c + 3 * T], s.v[c + 3 * T], y3);
      }
      for (; c <= r; c += T) y0 = fma(row[c], s.v[c], y0);
      for (; c + 3 * T < n; c += 4 * T) {
        y0 = fma(A[tri(c) + r], s.v[c], y0);
        y1 = fma(A[tri(c + T) + r], s.v[c + T], y1);
        y2 = fma(A[tri(c + 2 * T) + r], s.v[c + 2 * T], y2);
        y3 = fma(A[tri(c + 3 * T) + r], s.v[c + 3 * T], y3);
      }
      for (; c < n; c += T) y1 = fma(A[tri(c) + r], s.v[c], y1);
      y = (y0 + y1) + (y2 + y3);
    }
    for (int o = T >> 1; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
    y *= tau;
    const double vr = mine ? s.v[r] : 0.0;
    if (mine && k == 0) s.p[r] = y;
    const double a2 = -0.5 * tau * block_sum_alt(mine && k == 0 ? y * vr : 0.0, s.red, parity);
    // A22 -= v w^T + w v^T (w = p + a2 v) on the row segments, keeping the next column's norm part
    double part = 0.0;
    if (mine) {
      const double wr = y + a2 * vr;
      double* row = A + tr;
      int c = i + 1 + k;
      for (; c + 3 * T <= r; c += 4 * T) {
        const double v0 = s.v[c], v1 = s.v[c + T], v2 = s.v[c + 2 * T], v3 = s.v[c + 3 * T];
        const double w0 = s.p[c] + a2 * v0, w1 = s.p[c + T] + a2 * v1, w2 = s.p[c + 2 * T] + a2 * v2,
                     w3 = s.p[c + 3 * T] + a2 * v3;
        const double a0 = row[c], a1 = row[c + T], a2_ = row[c + 2 * T], a3 = row[c + 3 * T];
        row[c] = a0 - (vr * w0 + wr * v0);
        row[c + T] = a1 - (vr * w1 + wr * v1);
        row[c + 2 * T] = a2_ - (vr * w2 + wr * v2);
        row[c + 3 * T] = a3 - (vr * w3 + wr * v3);
      }
      for (; c <= r; c += T) {
        const double vc = s.v[c], wc = s.p[c] + a2 * vc;
        row[c] -= vr * wc + wr * vc;
      }
      if (k == 0 && r >= i + 3) {
        const double x = row[i + 1];
        part = x * x;
      }
    }
    xn2 = block_sum_alt(part, s.red, parity);
  }
  if (close && t == 0) {
    if (n >= 2) {
      s.d[n - 2] = A[tri(n - 2) + n - 2];
      s.e[n - 2] = A[tri(n - 1) + n - 2];
      s.tau[n - 2] = 0.0;
    }
    s.d[n - 1] = A[tri(n - 1) + n - 1];
    s.e[n - 1] = 0.0;
  }
  __syncthreads();
}

// Householder reduction of the packed n x n matrix A (shared or global memory).
__device__ __noinline__ void tridiagonalize(int n, double* __restrict__ A, const EigenScratch& s) {
  householder_columns(n, A, s.v, s.p, s.red, s.tau, s.e, s.d, n - 2, true);
}

// Sturm counts at M shifts at once, without divisions (see the ratio form above for the
// reference recurrence): p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2}; sign changes between
// consecutive values count the eigenvalues below x. Pairs are rescaled by powers of two every
// 8 steps (each step grows |p| by far less than 2^32 for the matrices here), exact for ratios.
template <int M>
__device__ __forceinline__ void sturm_multi(const double* __restrict__ d, const double* __restrict__ e2, int n,
                                            const double (&x)[M], double pivmin, int (&cnt)[M]) {
  (void)pivmin;
  constexpr double kBig = 0x1p256, kSmall = 0x1p-256;
  double p[M], pm[M];
  unsigned sg[M];
#pragma unroll
  for (int t = 0; t < M; ++t) {
    pm[t] = 1.0;
    p[t] = d[0] - x[t];
    sg[t] = __double_as_longlong(p[t]) < 0 ? 1u : 0u;
    cnt[t] = (int)sg[t];
  }
  int i = 1;
  for (; i + 8 <= n; i += 8) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const double di = d[i + u], ei = e2[i + u - 1];
#pragma unroll
      for (int t = 0; t < M; ++t) {
        const double pn = fma(di - x[t], p[t], -ei * pm[t]);
        const unsigned s = __double_as_longlong(pn) < 0 ? 1u : 0u;
        cnt[t] += (int)(s ^ sg[t]);
        sg[t] = s;
        pm[t] = p[t];
        p[t] = pn;
      }
    }
#pragma unroll
    for (int t = 0; t < M; ++t) {
      const double m = fmax(fabs(p[t]), fabs(pm[t]));
      const double sc = m > kBig ? kSmall : (m < kSmall ? kBig : 1.0);
      p[t] *= sc;
      pm[t] *= sc;
    }
  }
  for (; i < n; ++i) {
    const double di = d[i], ei = e2[i - 1];
#pragma unroll
    for (int t = 0; t < M; ++t) {
      const double pn = fma(di - x[t], p[t], -ei * pm[t]);
      const unsigned s = __double_as_longlong(pn) < 0 ? 1u : 0u;
      cnt[t] += (int)(s ^ sg[t]);
      sg[t] = s;
      pm[t] = p[t];
      p[t] = pn;
    }
  }
}

// Splits T where the coupling is negligible and computes the lowest `kval` eigenvalues.
// Leaves pivmin / tnorm in misc[0] / misc[1]. With `prev` (the same eigenvalues of the
// previous SCF iteration) and `dprev` (their last change) the search starts from a bracket
// around prev[j] once Sturm counts confirm it.
__device__ __noinline__ void tridiag_eigenvalues(int n, int kval, const EigenScratch& s_, const double* prev = nullptr,
                                    const double* dprev = nullptr) {
  struct {
    double *d, *e, *e2, *misc, *lam;
    int *blk, *nblk;
  } s = {s_.d, s_.e, s_.e2, s_.misc, s_.lam, s_.blk, s_.nblk};
  const int tid = threadIdx.x;
  constexpr double eps = 2.220446049250313e-16;
  if (tid == 0) {
    // Gershgorin bounds of the unsplit T, then split where |e_i| <= 1000 eps ||T||: an
    // absolute criterion, so exactly degenerate eigenvalues (which Householder leaves joined
    // by couplings of a few eps ||T||) land in separate blocks.
    double gl = s.d[0], gu = s.d[0];
    for (int i = 0; i < n; ++i) {
      const double rad = (i + 1 < n ? fabs(s.e[i]) : 0.0) + (i > 0 ? fabs(s.e[i - 1]) : 0.0);
      gl = fmin(gl, s.d[i] - rad);
      gu = fmax(gu, s.d[i] + rad);
    }
    const double tnorm = fmax(fabs(gl), fabs(gu));
    const double cut = 1000.0 * eps * tnorm;
    int nb = 0;
    s.blk[0] = 0;
    double emax = 0.0;
    for (int i = 0; i < n; ++i) {
      double ei = (i + 1 < n) ? s.e[i] : 0.0;
      if (i + 1 < n && fabs(ei) <= cut) {
        ei = 0.0;
        s.e[i] = 0.0;
        s.blk[++nb] = i + 1;
      }
      s.e2[i] = ei * ei;
      emax = fmax(emax, ei * ei);
    }
    s.blk[++nb] = n;
    *s.nblk = nb;
    s.misc[0] = 2.2250738585072014e-308 * fmax(1.0, emax);  // pivmin
    s.misc[1] = tnorm;
    s.misc[2] = gl - 4.0 * eps * tnorm * n - 1.0e-300;
    s.misc[3] = gu + 4.0 * eps * tnorm * n + 1.0e-300;
  }
  __syncthreads();
  const double pivmin = s.misc[0], tnorm = s.misc[1], glo = s.misc[2], ghi = s.misc[3];
  // Multisection: a group of g lanes (a power of two, g <= 32, kval * g <= kThreads) brackets
  // one eigenvalue; each step the group takes Sturm counts at P = g * kPts interior points (kPts
  // per lane, evaluated together), which cuts the bracket by P + 1 instead of 2.
  // Invariant: count(lo) <= j < count(hi).
  constexpr int kPts = 2;
  int g = 1;
  while (g < 32 && kval * (2 * g) <= kThreads) g *= 2;
  const int P = g * kPts;
  const int lane = tid & 31;
  const int gbase = lane & ~(g - 1), gl = lane & (g - 1);
  const unsigned gbits = g == 32 ? 0xffffffffu : ((1u << g) - 1u);
  for (int j0 = 0; j0 < kval; j0 += kThreads / g) {
    const int j = j0 + tid / g;
    const bool active = j < kval;
    double lo = glo, hi = ghi;
    if (prev) {
      // warm bracket around the previous SCF iteration's value, widened until two Sturm
      // counts confirm that it holds eigenvalue j (else the Gershgorin interval stays)
      const double c0 = active ? prev[j] : 0.0;
      const double w0 = active ? fmax(4.0 * fabs(dprev[j]), 1.0e-9 * fmax(tnorm, 1.0)) : 0.0;
      double x[4];
      int cn[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {  // brackets w0 and 64 w0: lower ends on even t, upper on odd
        const double w = w0 * (t >= 2 ? 64.0 : 1.0);
        x[t] = (t & 1) ? fmin(c0 + w, ghi) : fmax(c0 - w, glo);
      }
      if (active) sturm_multi<4>(s.d, s.e2, n, x, pivmin, cn);
      if (active) {
        if (x[0] < x[1] && cn[0] <= j && cn[1] >= j + 1) {
          lo = x[0];
          hi = x[1];
        } else if (x[2] < x[3] && cn[2] <= j && cn[3] >= j + 1) {
          lo = x[2];
          hi = x[3];
        }
      }
    }
    bool act = active;
    for (int it = 0; it < 128; ++it) {
      if (act) {
        const double mid = 0.5 * (lo + hi);
        if (hi - lo <= 2.0 * eps * fmax(fabs(lo), fabs(hi)) + 4.0 * pivmin || !(mid > lo && mid < hi)) act = false;
      }
      if (!__any_sync(0xffffffffu, act)) break;
      double x[kPts];
      int cn[kPts];
#pragma unroll
      for (int t = 0; t < kPts; ++t) x[t] = lo + (hi - lo) * (double)(gl * kPts + t + 1) / (double)(P + 1);
      if (act) sturm_multi<kPts>(s.d, s.e2, n, x, pivmin, cn);
      int tf = kPts;  // this lane's first point above eigenvalue j
#pragma unroll
      for (int t = kPts - 1; t >= 0; --t)
        if (act && cn[t] > j) tf = t;
      const unsigned bal = __ballot_sync(0xffffffffu, act && tf < kPts);
      const unsigned mine = (bal >> gbase) & gbits;
      const int src = mine ? gbase + __ffs(mine) - 1 : gbase;
      const int tsrc = __shfl_sync(0xffffffffu, tf, src);
      if (act) {
        double nlo, nhi;
        if (mine == 0u) {  // every point is at or below eigenvalue j
          nlo = lo + (hi - lo) * (double)P / (double)(P + 1);
          nhi = hi;
        } else {
          const int f = (src - gbase) * kPts + tsrc;  // first point above it
          nlo = f > 0 ? lo + (hi - lo) * (double)f / (double)(P + 1) : lo;
          nhi = lo + (hi - lo) * (double)(f + 1) / (double)(P + 1);
        }
        if (!(nhi - nlo < hi - lo)) act = false;
        else {
          lo = nlo;
          hi = nhi;
        }
      }
    }
    if (active && gl == 0) s.lam[j] = 0.5 * (lo + hi);
  }
  __syncthreads();
}

// Eigenvector j (< kvec) of T into Y[j*n .. j*n+n) (zero outside its block). `tf` is per-CTA
// global scratch of kvec * 6n doubles.
__device__ __noinline__ void tridiag_vectors(int n, int kvec, double* Y, double* tf, const EigenScratch& s_) {
  struct {
    const double *d, *e, *e2, *lam, *misc;
    const int *blk, *nblk;
    int* vinfo;
  } s = {s_.d, s_.e, s_.e2, s_.lam, s_.misc, s_.blk, s_.nblk, s_.vinfo};
  const int tid = threadIdx.x;
  const double pivmin = s.misc[0], tnorm = s.misc[1];
  const int nb = *s.nblk;
  const double win = 1.0e-11 * fmax(tnorm, 1.0);
  // Two halves of the CTA work on the same vectors: warps 0-3 (half 0) form the top-down
  // factorisation L+ D+ L+^T of T - lam, warps 4-7 (half 1) the bottom-up U- D- U-^T; both are
  // chains of divisions, so running them side by side halves the latency per vector. Then half 0
  // picks the twist index, and the halves fill the vector above and below it. Per-vector scratch
  // in tf (6 n): D+, L+, U-, D- (the pivots after clamping), then [twist, block], [norm parts].
  constexpr int kHalf = kThreads / 2;
  const int half = tid / kHalf, hj = tid % kHalf;
  for (int j = hj; j < kvec; j += kHalf) {
    const double lam = s.lam[j];
    // which unreduced block holds this eigenvalue (degenerate copies go to successive blocks);
    // an unsplit T (the usual case) has one block, and the three Sturm counts are not needed
    int pos = nb == 1 ? 0 : j - sturm(s.d, s.e2, 0, n - 1, lam - win, pivmin);
    int b = nb == 1 ? 0 : -1;
    for (int q = 0; q < nb && b < 0; ++q) {
      const int lo = s.blk[q], hi = s.blk[q + 1] - 1;
      const int c = sturm(s.d, s.e2, lo, hi, lam + win, pivmin) - sturm(s.d, s.e2, lo, hi, lam - win, pivmin);
      if (pos < c) b = q;
      else pos -= c;
    }
    if (b < 0) b = 0;  // inconsistent counts (not expected): block 0
    if (half == 0) s.vinfo[j] = b;
    const int lo = s.blk[b], hi = s.blk[b + 1] - 1, m = hi - lo + 1;
    double* y = Y + (size_t)j * n;
    for (int i = half; i < n; i += 2) y[i] = 0.0;
    if (m == 1) continue;
    double* Dp = tf + (size_t)j * 6 * n;
    double* Lp = Dp + n;
    double* Um = Lp + n;
    double* Dm = Um + n;
    if (half == 0) {  // T - lam = L+ D+ L+^T (top-down)
      double dp = s.d[lo] - lam;
      for (int i = 0; i < m - 1; ++i) {
        if (fabs(dp) < pivmin) dp = dp < 0.0 ? -pivmin : pivmin;
        Dp[i] = dp;
        const double ei = s.e[lo + i];
        Lp[i] = ei / dp;
        dp = (s.d[lo + i + 1] - lam) - Lp[i] * ei;
      }
      if (fabs(dp) < pivmin) dp = dp < 0.0 ? -pivmin : pivmin;
      Dp[m - 1] = dp;
    } else {  // T - lam = U- D- U-^T (bottom-up)
      double dm = s.d[hi] - lam;
      if (fabs(dm) < pivmin) dm = dm < 0.0 ? -pivmin : pivmin;
      Dm[m - 1] = dm;
      for (int i = m - 2; i >= 0; --i) {
        const double ei = s.e[lo + i];
        Um[i] = ei / dm;
        dm = (s.d[lo + i] - lam) - Um[i] * ei;
        if (fabs(dm) < pivmin) dm = dm < 0.0 ? -pivmin : pivmin;
        Dm[i] = dm;
      }
    }
  }
  __syncthreads();
  // twist index r minimising |gamma_i| = |D+_i + D-_i - (d_i - lam)| (the largest index among ties,
  // as a downward scan with a strict comparison finds it)
  if (half == 0)
    for (int j = hj; j < kvec; j += kHalf) {
      const double lam = s.lam[j];
      const int b = s.vinfo[j], lo = s.blk[b], hi = s.blk[b + 1] - 1, m = hi - lo + 1;
      if (m == 1) continue;
      double* Dp = tf + (size_t)j * 6 * n;
      const double* Dm = Dp + 3 * n;
      double best = fabs(Dp[m - 1] + Dm[m - 1] - (s.d[hi] - lam));
      int r = m - 1;
      for (int i = m - 2; i >= 0; --i) {
        const double g = fabs(Dp[i] + Dm[i] - (s.d[lo + i] - lam));
        if (g < best) {
          best = g;
          r = i;
        }
      }
      reinterpret_cast<int*>(Dp + 4 * n)[0] = r;
    }
  __syncthreads();
  // solve N_r D_r N_r^T y = gamma_r e_r: half 0 the rows above r, half 1 from r down; partial norms
  for (int j = hj; j < kvec; j += kHalf) {
    const int b = s.vinfo[j], lo = s.blk[b], hi = s.blk[b + 1] - 1, m = hi - lo + 1;
    double* y = Y + (size_t)j * n;
    double* Dp = tf + (size_t)j * 6 * n;
    if (m == 1) {
      if (half == 0) y[lo] = 1.0;
      continue;
    }
    const double* Lp = Dp + n;
    const double* Um = Lp + n;
    const int r = reinterpret_cast<const int*>(Dp + 4 * n)[0];
    double nrm = 0.0;
    if (half == 0) {
      double yn = 1.0, ynn = 0.0;  // y[lo + i + 1], y[lo + i + 2]
      for (int i = r - 1; i >= 0; --i) {
        double z = -Lp[i] * yn;
        if (yn == 0.0 && i + 2 < m) z = -(s.e[lo + i + 1] / s.e[lo + i]) * ynn;
        y[lo + i] = z;
        nrm = fma(z, z, nrm);
        ynn = yn;
        yn = z;
      }
    } else {
      y[lo + r] = 1.0;
      nrm = 1.0;
      double yc = 1.0, yp = 0.0;  // y[lo + i], y[lo + i - 1] (the latter read only after a zero)
      for (int i = r; i < m - 1; ++i) {
        double z = -Um[i] * yc;
        if (yc == 0.0 && i >= 1) z = -(s.e[lo + i - 1] / s.e[lo + i]) * yp;
        y[lo + i + 1] = z;
        nrm = fma(z, z, nrm);
        yp = yc;
        yc = z;
      }
    }
    Dp[5 * n + half] = nrm;
  }
  __syncthreads();
  for (int j = hj; j < kvec; j += kHalf) {
    const int b = s.vinfo[j], lo = s.blk[b], hi = s.blk[b + 1] - 1, m = hi - lo + 1;
    if (m == 1) continue;
    const double* Dp = tf + (size_t)j * 6 * n;
    const int r = reinterpret_cast<const int*>(Dp + 4 * n)[0];
    const double scale = 1.0 / sqrt(Dp[5 * n] + Dp[5 * n + 1]);
    double* y = Y + (size_t)j * n;
    if (half == 0)
      for (int i = lo; i < lo + r; ++i) y[i] *= scale;
    else
      for (int i = lo + r; i <= hi; ++i) y[i] *= scale;
  }
  __syncthreads();
  // Eigenvalues of one block closer than 1e-7 ||T||: the twisted vectors are not reliable
  // there, so every cluster member after the first is recomputed by inverse iteration on a
  // row-pivoted LU of T_b - lam, re-orthogonalised against the earlier members of its
  // cluster (the dstein scheme). One thread per block; clusters are rare.
  const double ctol = 1.0e-7 * fmax(tnorm, 1.0), tiny = 2.220446049250313e-16 * fmax(tnorm, 1.0);
  for (int b = tid; b < nb; b += kThreads) {
    const int lo = s.blk[b], hi = s.blk[b + 1] - 1, m = hi - lo + 1;
    int head = -1, prev = -1;
    for (int j = 0; j < kvec; ++j) {
      if (s.vinfo[j] != b) continue;
      if (prev < 0 || s.lam[j] - s.lam[prev] >= ctol) {
        head = j;
        prev = j;
        continue;
      }
      prev = j;
      double* dd = tf + (size_t)j * 6 * n;
      double* dl = dd + n;
      double* du = dl + n;
      double* du2 = du + n;
      double* pv = du2 + n;
      const double sg = s.lam[j];
      for (int i = 0; i < m; ++i) {
        dd[i] = s.d[lo + i] - sg;
        if (i + 1 < m) dl[i] = du[i] = s.e[lo + i];
      }
      for (int i = 0; i + 1 < m; ++i) {
        if (fabs(dd[i]) >= fabs(dl[i])) {
          if (dd[i] == 0.0) dd[i] = tiny;
          const double f = dl[i] / dd[i];
          dl[i] = f;
          dd[i + 1] -= f * du[i];
          if (i + 2 < m) du2[i] = 0.0;
          pv[i] = 0.0;
        } else {
          const double f = dd[i] / dl[i];
          dd[i] = dl[i];
          dl[i] = f;
          const double t = du[i];
          du[i] = dd[i + 1];
          dd[i + 1] = t - f * dd[i + 1];
          if (i + 2 < m) {
            du2[i] = du[i + 1];
            du[i + 1] = -f * du[i + 1];
          }
          pv[i] = 1.0;
        }
      }
      for (int i = 0; i < m; ++i)
        if (fabs(dd[i]) < tiny) dd[i] = dd[i] < 0.0 ? -tiny : tiny;
      double* x = Y + (size_t)j * n + lo;
      for (int i = 0; i < m; ++i) x[i] = sin(1.0 + 0.7 * i + 1.3 * j);
      for (int it = 0; it < 3; ++it) {
        for (int i = 0; i + 1 < m; ++i) {
          if (pv[i] == 0.0) {
            x[i + 1] -= dl[i] * x[i];
          } else {
            const double t = x[i];
            x[i] = x[i + 1];
            x[i + 1] = t - dl[i] * x[i];
          }
        }
        x[m - 1] /= dd[m - 1];
        if (m > 1) x[m - 2] = (x[m - 2] - du[m - 2] * x[m - 1]) / dd[m - 2];
        for (int i = m - 3; i >= 0; --i) x[i] = (x[i] - du[i] * x[i + 1] - du2[i] * x[i + 2]) / dd[i];
        for (int pass = 0; pass < 2; ++pass)
          for (int q = head; q < j; ++q) {
            if (s.vinfo[q] != b) continue;
            const double* yq = Y + (size_t)q * n + lo;
            double dot = 0.0;
            for (int i = 0; i < m; ++i) dot += yq[i] * x[i];
            for (int i = 0; i < m; ++i) x[i] -= dot * yq[i];
          }
        double nrm = 0.0;
        for (int i = 0; i < m; ++i) nrm += x[i] * x[i];
        nrm = 1.0 / sqrt(nrm);
        for (int i = 0; i < m; ++i) x[i] *= nrm;
      }
    }
  }
  __syncthreads();
}

// Y[j] <- H(0) H(1) ... H(n-3) Y[j] for j < kvec, two vectors per warp held in registers.
// One warp applies the reflectors to NV vectors at a time, RT rows per lane held in registers
// (n <= 32 RT). Per reflector the NV partial dot products are reduced together (their shuffle
// chains overlap), so the latency of a reflector is paid once for NV vectors.
template <int RT, int NV>
__device__ __forceinline__ void back_transform_t(int n, int kvec, const double* __restrict__ A, double* Y,
                                                 const double* __restrict__ tau_) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int j0 = NV * warp; j0 < kvec; j0 += NV * kWarps) {
    double z[NV][RT];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const double* y = Y + (size_t)(j0 + v < kvec ? j0 + v : j0) * n;
#pragma unroll
      for (int t = 0; t < RT; ++t) {
        const int r = lane + 32 * t;
        z[v][t] = r < n ? y[r] : 0.0;
      }
    }
    for (int i = n - 3; i >= 0; --i) {
      const double tau = tau_[i];
      if (tau == 0.0) continue;
      double vr[RT];
#pragma unroll
      for (int t = 0; t < RT; ++t) {
        const int r = lane + 32 * t;
        vr[t] = (r > i && r < n) ? (r == i + 1 ? 1.0 : A[tri(r) + i]) : 0.0;
      }
      double a[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        double acc = 0.0;
#pragma unroll
        for (int t = 0; t < RT; ++t) acc = fma(vr[t], z[v][t], acc);
        a[v] = acc;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int v = 0; v < NV; ++v) a[v] += __shfl_xor_sync(0xffffffffu, a[v], o);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const double s = a[v] * tau;
#pragma unroll
        for (int t = 0; t < RT; ++t) z[v][t] = fma(-s, vr[t], z[v][t]);
      }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      if (j0 + v >= kvec) break;
      double* y = Y + (size_t)(j0 + v) * n;
#pragma unroll
      for (int t = 0; t < RT; ++t) {
        const int r = lane + 32 * t;
        if (r < n) y[r] = z[v][t];
      }
    }
  }
  __syncthreads();
}

// The reflectors of column i (v_{i+1} = 1, v_r = A(r, i) below) applied from the last to the
// first. Up to n = 64 each lane holds 2 rows and a warp 4 vectors (the n/2 or so occupied vectors
// then keep all eight warps busy, which measured faster than 8 vectors on four warps).
__device__ __noinline__ void back_transform(int n, int kvec, const double* __restrict__ A, double* Y, const EigenScratch& s_) {
  if (n <= 64) back_transform_t<2, 4>(n, kvec, A, Y, s_.tau);
  else if (n <= 128) back_transform_t<4, 4>(n, kvec, A, Y, s_.tau);
  else back_transform_t<kRowT, 2>(n, kvec, A, Y, s_.tau);
}

// All eigenvalues of the saved tridiagonal (d, e) -- used once at the end for the MO energies.
__device__ __noinline__ void all_eigenvalues(int n, const double* d, const double* e, double* out, const EigenScratch& s) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < n; ++i) {
      s.d[i] = d[i];
      s.e[i] = e[i];
    }
  }
  __syncthreads();
  tight::tridiag_eigenvalues(n, n, s);
  for (int j = threadIdx.x; j < n; j += kThreads) out[j] = s.lam[j];
  __syncthreads();
}

// ------------------------------------------------------------------ job setup + H_core
__device__ __forceinline__ int psize(const Ctx& c, int a) { return heavy(c, a) ? 10 : 1; }

__device__ __noinline__ void setup_job(Ctx& c) {
  const KernelArgs& A = *c.A;
  const int tid = threadIdx.x;
  for (int a = tid; a < c.N; a += kThreads) {
    c.sz[a] = A.z[c.job.atom0 + a];
    for (int k = 0; k < 3; ++k) c.sxyz[3 * a + k] = A.xyz[3 * (size_t)(c.job.atom0 + a) + k];
  }
  c.W = c.Wg;
  __syncthreads();
  if (tid == 0) {
    int off = 0, pr = 0;
    for (int a = 0; a < c.N; ++a) {
      c.soff[a] = off;
      off += A.elem[c.sz[a]].norb;
      c.sprow[a] = pr;
      pr += psize(c, a);
    }
    c.sprow[c.N] = pr;
    int ro = 0;
    for (int a = 0; a < c.N; ++a) {
      c.sroff[a] = ro;
      ro += psize(c, a) * (pr - c.sprow[a + 1]);
    }
  }
  __syncthreads();
}

// H_core (hamiltonian.rs:191-344) and the pair table W (pair (u < v), blocks in (a, b) orientation, row-major); returns the
// core-core energy (repulsion.rs:13-27) to every thread.
__device__ __noinline__ double build_core(Ctx& c) {
  const KernelArgs& A = *c.A;
  const int n = c.n, N = c.N, tid = threadIdx.x;
  double* hacc = c.jacc;  // [N*10] diagonal-block accumulators
  for (int k = tid; k < N * 10; k += kThreads) hacc[k] = 0.0;
  __syncthreads();
  double ecc = 0.0;
  const int npairs = N * (N - 1) / 2;
  for (int t = tid; t < npairs; t += kThreads) {
    int u, v;
    pair_uv(N, t, u, v);
    const bool hu = heavy(c, u), hv = heavy(c, v);
    const int a = (hu || !hv) ? u : v, b = a == u ? v : u;
    double* w = c.W + c.sroff[u] + psize(c, u) * (c.sprow[v] - c.sprow[u + 1]);
    ecc += core_pair<true>(A.elem[c.sz[a]], A.elem[c.sz[b]], A.elem[c.sz[u]], A.elem[c.sz[v]], *A.pairs, c.sxyz + 3 * a,
                           c.sxyz + 3 * b, c.soff[a], c.soff[b], (size_t)n, hacc + a * 10, hacc + b * 10, w, 1, c.H);
  }
  __syncthreads();
  // diagonal blocks: U + sum of electron-core attractions
  for (int k = tid; k < N * 16; k += kThreads) {
    const int a = k >> 4, mu = (k >> 2) & 3, nu = k & 3;
    const ElemDev& e = A.elem[c.sz[a]];
    if (mu >= e.norb || nu >= e.norb) continue;
    double h = hacc[a * 10 + pk(mu, nu)];
    if (mu == nu) h += mu == 0 ? e.uss : e.upp;
    c.H[(size_t)(c.soff[a] + mu) * n + c.soff[a] + nu] = h;
  }
  __syncthreads();
  return block_sum(ecc, c.red);
}

// ------------------------------------------------------------------------ Fock build
// Coulomb part of one atom pair (fock.rs:106-159): J_a[p] += sum_q W[p][q] Pb_q, J_b[q] += sum_p Pa_p W[p][q].
template <int NA, int NB>
__device__ __forceinline__ void coulomb_pair(int a, int b, const double* __restrict__ dpk, double* jacc,
                                             const double* __restrict__ w) {
  constexpr int PA = NA == 4 ? 10 : 1, PB = NB == 4 ? 10 : 1;
  double db[PB], jb[PB];
#pragma unroll
  for (int q = 0; q < PB; ++q) {
    db[q] = dpk[b * 10 + q];
    jb[q] = 0.0;
  }
#pragma unroll
  for (int p = 0; p < PA; ++p) {
    const double da = dpk[a * 10 + p];
    double acc = 0.0;
#pragma unroll
    for (int q = 0; q < PB; ++q) {
      const double wv = w[p * PB + q];
      acc = fma(db[q], wv, acc);
      jb[q] = fma(da, wv, jb[q]);
    }
    atomicAdd(&jacc[a * 10 + p], acc);
  }
#pragma unroll
  for (int q = 0; q < PB; ++q) atomicAdd(&jacc[b * 10 + q], jb[q]);
}

template <int NA, int NB>
__device__ __forceinline__ void fock_item(bool uhf, int n, int a, int b, int oa, int ob, const double* __restrict__ dpk, double* jacc,
                                          const double* __restrict__ H, const double* __restrict__ w, const double* Pt,
                                          const double* Pa, const double* Pb, double* F, double* G) {
  coulomb_pair<NA, NB>(a, b, dpk, jacc, w);
  if (uhf) fock_pair<NA, NB, true>(n, oa, ob, H, w, Pt, Pa, Pb, F, G);
  else fock_pair<NA, NB, false>(n, oa, ob, H, w, Pt, Pa, Pb, F, G);
}

// F = H + J(Pt) - K(Ps) (fock.rs:285-332). Pt = total density; for RHF Ps = Pt / 2 (Pb null),
// for UHF two spin Focks F (from Pa) and G (from Pb) are built in one pass.
__device__ __noinline__ void build_fock(Ctx& c, const double* Pt, const double* Pa, const double* Pb, double* F, double* G) {
  const KernelArgs& A = *c.A;
  const int n = c.n, N = c.N, tid = threadIdx.x;
  const bool uhf = Pb != nullptr;
  // packed atomic densities (fock.rs:93-100); the Coulomb accumulators start at zero
  for (int k = tid; k < N * 10; k += kThreads) {
    const int a = k / 10, p = k % 10;
    const int no = A.elem[c.sz[a]].norb;
    c.jacc[k] = 0.0;
    double v = 0.0;
    if (no == 4 || p == 0) {
      int hi, lo;
      unpk(p, hi, lo);
      const int oa = c.soff[a];
      v = Pt[(size_t)(oa + hi) * n + oa + lo];
      if (hi != lo) v *= 2.0;
    }
    c.dpk[k] = v;
  }
  __syncthreads();
  const int npairs = N * (N - 1) / 2;
  {
    const int* __restrict__ sprow = c.sprow;
    const int* __restrict__ soff = c.soff;
    const int* __restrict__ sroff = c.sroff;
    const double* __restrict__ W = c.W;
    const double* __restrict__ H = c.H;
    const double* __restrict__ dpk = c.dpk;
    double* jacc = c.jacc;
    for (int t = tid; t < npairs; t += kThreads) {
      int u, v;
      pair_uv(N, t, u, v);
      const int su = sprow[u + 1] - sprow[u], sv = sprow[v + 1] - sprow[v];  // packed sizes: 10 sp, 1 s
      const bool hu = su == 10, hv = sv == 10;
      const int a = (hu || !hv) ? u : v, b = a == u ? v : u;
      const double* w = W + sroff[u] + su * (sprow[v] - sprow[u + 1]);
      const int oa = soff[a], ob = soff[b];
      if (hu && hv) fock_item<4, 4>(uhf, n, a, b, oa, ob, dpk, jacc, H, w, Pt, Pa, Pb, F, G);
      else if (hu || hv) fock_item<4, 1>(uhf, n, a, b, oa, ob, dpk, jacc, H, w, Pt, Pa, Pb, F, G);
      else fock_item<1, 1>(uhf, n, a, b, oa, ob, dpk, jacc, H, w, Pt, Pa, Pb, F, G);
    }
  }
  __syncthreads();
  // atom-diagonal blocks: H + one-centre J - K (fock.rs:244-282) + two-centre J
  for (int k = tid; k < N * 16; k += kThreads) {
    const int a = k >> 4, mu = (k >> 2) & 3, nu = k & 3;
    const ElemDev& e = A.elem[c.sz[a]];
    const int no = e.norb;
    if (mu >= no || nu >= no) continue;
    const int oa = c.soff[a];
    double ja = 0.0, ka = 0.0, kb = 0.0;
    for (int la = 0; la < no; ++la)
      for (int si = 0; si < no; ++si) {
        const double coul = oc_integral(e, mu, nu, la, si), exch = oc_integral(e, mu, la, nu, si);
        const size_t ix = (size_t)(oa + la) * n + oa + si;
        ja = fma(Pt[ix], coul, ja);
        if (uhf) {
          ka = fma(Pa[ix], exch, ka);
          kb = fma(Pb[ix], exch, kb);
        } else {
          ka = fma(0.5 * Pt[ix], exch, ka);
        }
      }
    const size_t ix = (size_t)(oa + mu) * n + oa + nu;
    const double base = c.H[ix] + c.jacc[a * 10 + pk(mu, nu)] + ja;
    F[ix] = base - ka;
    if (uhf) G[ix] = base - kb;
  }
  __syncthreads();
}

// The Fock matrices of a density (spin densities P, Q; the restricted one P alone) and the electronic energy to all
// threads. `sum`: n^2 doubles for P + Q.
__device__ __noinline__ double fock_energy(Ctx& c, bool uhf, const double* P, const double* Q, double* sum, double* F, double* G) {
  const int tid = threadIdx.x;
  const size_t nn = (size_t)c.n * c.n;
  double part = 0.0;
  if (!uhf) {
    tight::build_fock(c, P, nullptr, nullptr, F, nullptr);
    for (size_t k = tid; k < nn; k += kThreads) part = fma(P[k], c.H[k] + F[k], part);
  } else {
    for (size_t k = tid; k < nn; k += kThreads) sum[k] = P[k] + Q[k];
    __syncthreads();
    tight::build_fock(c, sum, P, Q, F, G);
    for (size_t k = tid; k < nn; k += kThreads) part += sum[k] * c.H[k] + P[k] * F[k] + Q[k] * G[k];
  }
  return 0.5 * block_sum(part, c.red);
}

// E = F P - P F into E (scf.rs:1039-1054): one GEMM, then antisymmetrise in place.
__device__ __noinline__ void commutator(Ctx& c, const double* Fm, const double* Pm, double* E) {
  const int n = c.n;
  cta_gemm<false>(n, n, n, 1.0, Fm, n, Pm, n, c.tile, false,
                         [&](int i, int j, double v) { E[(size_t)i * n + j] = v; });
  for (int k = threadIdx.x; k < n * n; k += kThreads) {
    const int i = k / n, j = k % n;
    if (j < i) {
      const double lo = E[(size_t)i * n + j], up = E[(size_t)j * n + i];
      E[(size_t)i * n + j] = lo - up;
      E[(size_t)j * n + i] = up - lo;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += kThreads) E[(size_t)i * n + i] = 0.0;
  __syncthreads();
}

// A-DIIS weights on the simplex by projected gradient (scf.rs:1152-1172, 1637-1693), one warp:
// lane k owns weight c_k and its gradient component; the Euclidean projection onto the simplex
// sorts the trial point (descending, ties by index, as a stable insertion sort does) and every
// lane runs the reference's serial cumulative-sum scan over the sorted values, so the weights are
// the ones the serial loop produces. `sm` is shared scratch of kMaxDepth * (2 kMaxDepth + 1) doubles.
__device__ __noinline__ void adiis_coeffs_warp(int m, const double* mg, double* out, double* sm) {
  constexpr int K = kMaxDepth;
  const int k = threadIdx.x & 31;
  const int last = m - 1;
  const double mnn = mg[last * K + last];
  double* S = sm;           // [K][K]
  double* T = sm + K * K;   // [K][K] S + S^T, the gradient's matrix (same sums as the reference's)
  double* d = T + K * K;    // [K]
  if (k < m) {
    d[k] = mg[k * K + last] - mnn;
    for (int j = 0; j < m; ++j) S[k * K + j] = mg[k * K + j] - mg[k * K + last] - mg[last * K + j] + mnn;
  }
  __syncwarp();
  if (k < m)
    for (int j = 0; j < m; ++j) T[k * K + j] = S[k * K + j] + S[j * K + k];
  __syncwarp();
  double L = 1.0e-12;
  for (int i = 0; i < m; ++i) {
    double row = 0.0;
    for (int j = 0; j < m; ++j) row += fabs(T[i * K + j]);
    L = fmax(L, row);
  }
  const double lr = 1.0 / L;
  // Every lane runs the whole iteration on the full state in registers (the lanes agree), so the
  // loop needs no shuffles: gradient, trial point, its stable descending order, the reference's
  // cumulative-sum scan for the simplex projection, and the change.
  double c[K];
#pragma unroll
  for (int j = 0; j < K; ++j) c[j] = j == last ? 1.0 : 0.0;
  for (int it = 0; it < 400; ++it) {
    double t[K];
#pragma unroll
    for (int q = 0; q < K; ++q) {
      double g = 2.0 * d[q < m ? q : 0];
#pragma unroll
      for (int j = 0; j < K; ++j)
        if (j < m) g += T[q * K + j] * c[j];
      t[q] = q < m ? c[q] - lr * g : 0.0;
    }
    // the trial point sorted descending by a 19-comparator network on a copy (unused entries
    // -inf, so they sort last); ties give equal values in either order, so the cumulative sums,
    // and with them the projection, are those of the reference's stable sort
    double u[K];
#pragma unroll
    for (int q = 0; q < K; ++q) u[q] = q < m ? t[q] : -INFINITY;
    constexpr int kNet[19][2] = {{0, 2}, {1, 3}, {4, 6}, {5, 7}, {0, 4}, {1, 5}, {2, 6}, {3, 7}, {0, 1}, {2, 3},
                                 {4, 5}, {6, 7}, {2, 4}, {3, 5}, {1, 4}, {3, 6}, {1, 2}, {3, 4}, {5, 6}};
#pragma unroll
    for (int e = 0; e < 19; ++e) {
      const double a = u[kNet[e][0]], b = u[kNet[e][1]];
      u[kNet[e][0]] = fmax(a, b);
      u[kNet[e][1]] = fmin(a, b);
    }
    double css = 0.0, theta = 0.0;
#pragma unroll
    for (int p = 0; p < K; ++p) {
      if (p >= m) break;
      css += u[p];
      const double tt = (css - 1.0) / (double)(p + 1);
      if (u[p] - tt > 0.0) theta = tt;
    }
    double delta = 0.0;
#pragma unroll
    for (int q = 0; q < K; ++q) {
      if (q >= m) break;
      const double pq = fmax(t[q] - theta, 0.0);
      delta += fabs(pq - c[q]);
      c[q] = pq;
    }
    if (delta < 1.0e-12) break;
  }
  if (k < m) {
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (q == k) out[k] = c[q];
  }
  __syncwarp();
}

// One iteration's accelerator step (scf.rs:1065-1173, 1240-1259, 1398-1413): the density joins the history, the new Gram row
// against the surviving entries and the new diagonal, then the CDIIS (thread 0) or A-DIIS (warp 0) weights of len + 1
// entries to c.coef. Returns whether they are usable.
__device__ __noinline__ bool diis_step(Ctx& c, bool uhf, bool keep, int len, int head, int depth, int slot_mats, const double* Fa,
                          const double* Ea, const double* Eb, double* Dh, const double* Pc) {
  const JobDesc& J = c.job;
  const int n = c.n, tid = threadIdx.x;
  const size_t nn = (size_t)n * n;
  if (keep)
    for (size_t k = tid; k < nn; k += kThreads) Dh[k] = Pc[k];
  __syncthreads();
  double acc[3 * kMaxDepth + 2];
#pragma unroll
  for (int q = 0; q < 3 * kMaxDepth + 2; ++q) acc[q] = 0.0;
  // Every product pairs two symmetric (F, D) or two antisymmetric (E) matrices: the diagonal plus twice the strict lower
  // triangle. Rows go to warps, columns to lanes.
  for (int r = tid >> 5; r < n; r += kWarps)
    for (int col = tid & 31; col <= r; col += 32) {
      const size_t k = (size_t)r * n + col;
      const double wgt = col == r ? 1.0 : 2.0;
      const double ea = Ea[k], fa = Fa[k];
      const double eb = uhf ? Eb[k] : 0.0;
      const double dn = keep ? Dh[k] : 0.0;
      double ee = ea * ea;
      if (uhf) ee = fma(eb, eb, ee);
      acc[3 * kMaxDepth] = fma(wgt, ee, acc[3 * kMaxDepth]);
      if (keep) acc[3 * kMaxDepth + 1] = fma(wgt, dn * fa, acc[3 * kMaxDepth + 1]);
#pragma unroll
      for (int l = 0; l < kMaxDepth; ++l) {
        if (l < len) {
          const double* bl = c.hist + (size_t)((head + l) % depth) * slot_mats * nn;
          double v = bl[nn + k] * ea;
          if (uhf) v = fma(bl[3 * nn + k], eb, v);
          acc[l] = fma(wgt, v, acc[l]);
          if (keep) {
            acc[kMaxDepth + l] = fma(wgt, dn * bl[k], acc[kMaxDepth + l]);                   // <D_new, F_l>
            acc[2 * kMaxDepth + l] = fma(wgt, bl[2 * nn + k] * fa, acc[2 * kMaxDepth + l]);  // <D_l, F_new>
          }
        }
      }
    }
  block_sums<3 * kMaxDepth + 2>(acc, c.red, c.misc);
  if (tid == 0) {
    for (int l = 0; l < len; ++l) {
      c.bg[l * kMaxDepth + len] = c.misc[l];
      c.bg[len * kMaxDepth + l] = c.misc[l];
      c.mg[len * kMaxDepth + l] = c.misc[kMaxDepth + l];
      c.mg[l * kMaxDepth + len] = c.misc[2 * kMaxDepth + l];
    }
    c.bg[len * kMaxDepth + len] = c.misc[3 * kMaxDepth];
    c.mg[len * kMaxDepth + len] = c.misc[3 * kMaxDepth + 1];
    const int m = len + 1;
    bool ok;
    int mode = 0;
    if (!uhf && J.accel == 2 && sqrt(c.misc[3 * kMaxDepth]) > J.adiis_switch) {
      ok = keep && m >= 2;
      mode = ok ? 1 : 0;
    } else {
      ok = cdiis_coeffs(m, c.bg, c.coef);
    }
    c.iv[0] = ok ? 1 : 0;
    c.iv[1] = mode;
  }
  __syncthreads();
  if (c.iv[1] == 1) {  // uniform across the CTA
    if (tid < 32) tight::adiis_coeffs_warp(len + 1, c.mg, c.coef, c.red);
    __syncthreads();
  }
  return c.iv[0] != 0;
}

// ------------------------------------------------------------------- eigensolve + density
// Diagonalises `in`: kval lowest eigenvalues into lam_out, kvec eigenvectors into Y (rows). The tridiagonal (d, e) is saved
// to `tri_save` (2n) for the final MO energies.
// With `warm`, lam_out holds the same eigenvalues from the previous SCF iteration and `dlam`
// their last change; both seed the eigenvalue search and are updated. Without it dlam is reset.
__device__ __noinline__ void eigensolve(Ctx& c, const SymInput& in, int kval, int kvec, double* Y, double* lam_out, double* tri_save,
                           bool warm = false, double* dlam = nullptr) {
  const int n = c.n;
  double* Ap = n <= c.A->sm.nsm ? c.tile : c.Ag;
  // rows to warps, columns to lanes (coalesced reads)
  for (int r = threadIdx.x >> 5; r < n; r += kWarps)
    for (int col = threadIdx.x & 31; col <= r; col += 32) {
      const size_t ix = (size_t)r * n + col;
      double v;
      if (in.len) {
        v = 0.0;
        for (int l = 0; l < in.len; ++l) v = fma(in.coef[l], in.hist[(size_t)((in.head + l) % in.depth) * in.stride + ix], v);
      } else {
        v = in.X[ix];
      }
      if (in.shift != 0.0) v += in.shift * ((r == col ? 1.0 : 0.0) - in.proj[ix]);
      Ap[tri(r) + col] = v;
    }
  __syncthreads();
  mark(c, kPhPack);
  tight::tridiagonalize(n, Ap, c.es);
  if (tri_save && threadIdx.x == 0)
    for (int i = 0; i < n; ++i) {
      tri_save[i] = c.es.d[i];
      tri_save[n + i] = c.es.e[i];
    }
  mark(c, kPhTridiag);
  const bool seeded = warm && dlam != nullptr;
  tight::tridiag_eigenvalues(n, kval, c.es, seeded ? lam_out : nullptr, seeded ? dlam : nullptr);
  for (int j = threadIdx.x; j < kval; j += kThreads) {
    if (dlam) dlam[j] = seeded ? c.es.lam[j] - lam_out[j] : 1.0e30;
    lam_out[j] = c.es.lam[j];
  }
  mark(c, kPhEigval);
  if (kvec > 0) {
    tight::tridiag_vectors(n, kvec, Y, c.tf, c.es);
    mark(c, kPhEigvec);
    tight::back_transform(n, kvec, Ap, Y, c.es);
  }
  __syncthreads();
  mark(c, kPhBack);
}

// Pnew = w Y^T Y (first k rows of Y); returns sum (Pnew - Pold)^2 to all threads. With
// damping lam > 0 the stored value is (1-lam) Pnew + lam Pold (scf.rs:1440-1448); the RMS
// uses the undamped Pnew, as the reference does.
__device__ __noinline__ double density(Ctx& c, const double* Y, int k, double w, const double* Pold, double* Pnew, double damp) {
  const int n = c.n;
  double sq = 0.0;
  if (k == 0) {
    for (int q = threadIdx.x; q < n * n; q += kThreads) {
      const double o = Pold[q];
      sq += o * o;
      Pnew[q] = damp > 0.0 ? damp * o : 0.0;
    }
    __syncthreads();
    return block_sum(sq, c.red);
  }
  cta_gemm<true>(n, n, k, w, Y, n, Y, n, c.tile, true, [&](int i, int j, double v) {
    if (i < j) return;
    const size_t ij = (size_t)i * n + j, ji = (size_t)j * n + i;
    const double o = Pold[ij];
    const double dlt = v - o;
    sq += (i == j ? 1.0 : 2.0) * dlt * dlt;
    const double st = damp > 0.0 ? (1.0 - damp) * v + damp * o : v;
    Pnew[ij] = st;
    Pnew[ji] = st;
  });
  return block_sum(sq, c.red);
}

}  // namespace tight
}  // namespace pm3gpu
