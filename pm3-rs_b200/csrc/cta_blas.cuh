// CTA-level building blocks: reductions and the symmetric-form FP64 products of the
// per-molecule SCF (commutator F P - P F and the density C_occ C_occ^T).
#pragma once
#include <cuda_runtime.h>

namespace pm3gpu {

constexpr int kThreads = 256;  // threads per SCF CTA
constexpr int kWarps = kThreads / 32;

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sum of `v` over the CTA; every thread gets the result. `red` needs kWarps doubles.
__device__ __forceinline__ double block_sum(double v, double* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double t = 0.0;
#pragma unroll
  for (int i = 0; i < kWarps; ++i) t += red[i];
  return t;
}
__device__ __forceinline__ double block_max(double v, double* red) {
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double t = red[0];
#pragma unroll
  for (int i = 1; i < kWarps; ++i) t = fmax(t, red[i]);
  return t;
}
// Several sums at once: v[0..K) per thread -> out[0..K) (in shared memory, visible to all
// threads after return). `red` needs K * kWarps doubles.
template <int K>
__device__ __forceinline__ void block_sums(double (&v)[K], double* red, double* out) {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < K; ++k) v[k] = warp_sum(v[k]);
  __syncthreads();
  if (l == 0) {
#pragma unroll
    for (int k = 0; k < K; ++k) red[k * kWarps + w] = v[k];
  }
  __syncthreads();
  if (threadIdx.x < K) {
    double t = 0.0;
    for (int i = 0; i < kWarps; ++i) t += red[threadIdx.x * kWarps + i];
    out[threadIdx.x] = t;
  }
  __syncthreads();
}

// Sums 32 values over the warp, lane l ending with the total of value l: 31 shuffles (5 per value when summed one by one).
__device__ __forceinline__ double warp_sum32(double (&v)[32]) {
  const int l = threadIdx.x & 31;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < o; ++k) {
      const double send = (l & o) ? v[k] : v[k + o], keep = (l & o) ? v[k + o] : v[k];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  return v[0];
}

__device__ __forceinline__ void cp_async8(double* dst, const double* src, bool in) {  // zero when !in
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int bytes = in ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mma_f64(double (&c)[4], const double (&a)[4], double b0, double b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}

// Lower triangle of an n x n product of symmetric form on the FP64 tensor instructions, k summed over K:
//   kComm:  C_ij = sum_k A_ik B_jk - B_ik A_jk   (A, B symmetric, row-major n x n, K = n)
//   else:   C_ij = sum_k A_ki A_kj               (A row-major K x n)
// A stage of 8 k-values of every row passes through shared memory once for all blocks (8-byte asynchronous copies, two
// stages in flight), and the warps keep 16 x 16 blocks of the lower triangle in registers, five each: one pass up to
// n = 128, two up to 176. Shared layout [k / 4][row][4]: the half-warps' fragment loads are 16 consecutive doubles. `sh`: lower_scratch(n) doubles.
// Each element goes through epi(i, j, value), i >= j. What bounds it: FP64 issue (n^3 / 64 cycles for the commutator).
__host__ __device__ constexpr int lower_scratch(int n, bool comm) { return 2 * 8 * ((n + 15) / 16 * 16) * (comm ? 2 : 1); }
template <bool kComm, class Epi>
__device__ __forceinline__ void lower_product(int n, int K, const double* __restrict__ A, const double* __restrict__ B,
                                              double* sh, Epi epi) {
  constexpr int kOwn = 5;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tg = lane & 3;
  const int nb = (n + 15) / 16, M = 16 * nb, blocks = nb * (nb + 1) / 2;
  const int stage = 8 * M * (kComm ? 2 : 1);  // doubles of one stage: A, then B
  const int steps = (K + 7) / 8;
  auto fill = [&](int st) {
    double* dst = sh + (st & 1) * stage;
    const int k0 = 8 * st;
    if (kComm) {  // rows of 8 consecutive values
      for (int e = tid; e < 8 * M; e += kThreads) {
        const int r = e >> 3, k = e & 7;
        const bool in = r < n && k0 + k < K;
        const int at = ((k >> 2) * M + r) * 4 + (k & 3), ix = in ? r * n + k0 + k : 0;
        cp_async8(dst + at, A + ix, in);
        cp_async8(dst + 8 * M + at, B + ix, in);
      }
    } else {  // one warp a k-value
      const int k = warp;
      for (int r = lane; r < M; r += 32) {
        const bool in = r < n && k0 + k < K;
        cp_async8(dst + ((k >> 2) * M + r) * 4 + (k & 3), A + (in ? (k0 + k) * n + r : 0), in);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int first = 0; first < blocks; first += kWarps * kOwn) {
    double acc[kOwn][2][4];
    int bi[kOwn], bj[kOwn];
#pragma unroll
    for (int q = 0; q < kOwn; ++q) {
      const int t = first + warp + kWarps * q;
      int I = (int)((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
      while (I * (I + 1) / 2 > t) --I;
      while ((I + 1) * (I + 2) / 2 <= t) ++I;
      bi[q] = t < blocks ? I : -1;
      bj[q] = t - I * (I + 1) / 2;
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[q][h][e] = 0.0;
    }
    fill(0);
    for (int st = 0; st < steps; ++st) {
      if (st + 1 < steps) {
        fill(st + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      __syncthreads();
      const double* __restrict__ sa = sh + (st & 1) * stage;
      const double* __restrict__ sb = sa + 8 * M;
#pragma unroll
      for (int q = 0; q < kOwn; ++q) {
        if (bi[q] < 0) continue;  // uniform in the warp
        const int ri = (16 * bi[q] + g) * 4 + tg, rj = (16 * bj[q] + g) * 4 + tg;
        const double af[4] = {sa[ri], sa[ri + 32], sa[4 * M + ri], sa[4 * M + ri + 32]};
        if (kComm) {
          const double pf[4] = {sb[ri], sb[ri + 32], sb[4 * M + ri], sb[4 * M + ri + 32]};
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            mma_f64(acc[q][h], af, sb[rj + 32 * h], sb[4 * M + rj + 32 * h]);
            mma_f64(acc[q][h], pf, -sa[rj + 32 * h], -sa[4 * M + rj + 32 * h]);
          }
        } else {
#pragma unroll
          for (int h = 0; h < 2; ++h) mma_f64(acc[q][h], af, sa[rj + 32 * h], sa[4 * M + rj + 32 * h]);
        }
      }
      __syncthreads();  // this stage is filled again next
    }
#pragma unroll
    for (int q = 0; q < kOwn; ++q) {
      if (bi[q] < 0) continue;
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = 16 * bi[q] + g + 8 * (e >> 1), j = 16 * bj[q] + 8 * h + 2 * tg + (e & 1);
          if (i < n && j <= i) epi(i, j, acc[q][h][e]);
        }
    }
  }
  __syncthreads();
}

}  // namespace pm3gpu
