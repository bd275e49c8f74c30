// Symmetric eigensolver for one matrix per CTA (n <= kMaxN), replacing the reference's faer
// `self_adjoint_eigen` (pm3-rs src/linalg.rs:221-263) on the SCF path:
//   1. Householder reduction to tridiagonal form with the matrix in registers (`tridiagonalize`).
//      The reflectors go to global memory, one row of `V` per reduced column.
//   2. Eigenvalues of the tridiagonal T by Sturm-count multisection, a group of lanes per
//      eigenvalue, started from the previous SCF iteration's eigenvalues when given.
//   3. Eigenvectors of T by twisted (N_r D_r N_r^T) factorisation, one thread per vector,
//      on the unreduced block holding the eigenvalue (T is split where |e_i| <= 1000 eps ||T||,
//      which separates exact degeneracies); members of a within-block cluster (gap below
//      1e-7 ||T||) after the first are redone by inverse iteration with re-orthogonalisation.
//   4. Back-transformation Z = Q Y, a group of lanes per 1 to 3 vectors held in registers, the
//      reflectors staged through shared memory.
// Only the eigenpairs the SCF needs are formed (the occupied block, plus one more value for
// the frontier gap). Eigenvalues come out ascending, as the reference requires.
#pragma once
#include <type_traits>

#include "cta_blas.cuh"

namespace pm3gpu {

constexpr int kMaxN = 256;          // largest basis handled by the per-CTA path

// The same shared-memory address, expressed from the shared window so that the compiler emits shared
// accesses: the scratch pointers reach these functions through memory, where their address space is lost, and
// generic loads and stores cost more (a reduced column of a 112 x 112 matrix 3.5k cycles against 2.4k).
template <class T>
__device__ __forceinline__ T* in_shared(T* p) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int off = (int)__cvta_generic_to_shared(p) - (int)__cvta_generic_to_shared(smem);
  return reinterpret_cast<T*>(smem + off);
}

struct EigenScratch {
  double* d;     // [n] diagonal of T
  double* e;     // [n] off-diagonal of T (e[i] couples i, i+1); zeroed where T splits
  double* e2;    // [n] e^2
  double* tau;   // [n] reflector scales
  double* v;     // [n] eigenvector scratch (norm parts)
  double* p;     // [n] eigenvector scratch (norm parts)
  double* lam;   // [n] eigenvalues (ascending)
  int* blk;      // [n+1] block starts (blk[0] = 0, ..., blk[nb] = n)
  int* nblk;     // [1]
  int* vinfo;    // [n] per eigenvector: its block index, and the twist index in the upper 16 bits
  double* red;   // reduction scratch (>= 8 * kWarps)
  double* misc;  // [8] broadcast scalars
  double* sh;    // shared scratch: reduction vectors, then memory blocks, then staged reflectors
  int sh_doubles;
};

// ---------------------------------------------------------------- 1. tridiagonalisation
// Householder reduction with the matrix in registers. The matrix sits at the end of a frame of
// 16 x 16 blocks (rows padded in front, so the columns retire from the first block on); thread
// (ty, tx) of the 16 x 16 thread grid owns element (16 I + ty, 16 J + tx) of every lower block
// (I >= J; a diagonal block holds both triangles). The last kRegB block columns live in registers;
// the block columns before them (n > 16 kRegB only) live in private memory slots, shared memory
// first, and are reduced by the same steps.
// The reflector of column i is H = I - tau v v^T with v = x - beta e_{i+1}, x the column below the diagonal
// (not scaled to v_{i+1} = 1): then A v = A x - beta A e_{i+1}, and the product A x needs neither the norm
// nor the square root and division that beta and tau take, which overlap with it.
// Two barriers per column. Between them one thread per row adds up the row's and the column
// partial sums of A x, forms w, and applies the column's update to the next column in advance (its
// old values were published with the partial sums), so that the next reflector is known when the
// rest of the matrix is updated.
// What bounds it: latency, the chain of two barriers, shuffles and shared-memory round trips that 8 warps a CTA do not hide:
// about 1500 cycles a column up to n = 64 or so; at n = 112 2.2k alone and 3.0k with two CTAs on the SM, where the four
// FMAs an element and column are 131 cycles of the FP64 pipe (5.8 % busy over a launch). Beyond 112 the memory blocks' traffic adds to it
// (n = 148: 4.9k).
constexpr int kRegB = 7;                        // block columns held in registers: 28 values a thread
constexpr int kRegRows = 16 * kRegB;
__host__ __device__ constexpr int frame_rows(int n) { return n <= kRegRows ? kRegRows : (n + 15) / 16 * 16; }
// doubles of shared scratch `tridiagonalize` needs for bases up to n (vectors; memory blocks go after them)
__host__ __device__ constexpr int tri_scratch(int n) { return 15 * frame_rows(n); }
// the same with every memory block in shared memory: kThreads doubles for each of the (nb - J) blocks of the columns J < nb - kRegB
__host__ __device__ constexpr int tri_resident(int n) {
  const int nb = frame_rows(n) / 16, mb = nb - kRegB;
  return tri_scratch(n) + kThreads * (mb * nb - mb * (mb - 1) / 2);
}

constexpr int kPart = 10;
struct TriCtx {
  double *xs, *vs, *ws, *raw, *rsum;  // [M] each
  double *cpart;                      // [M][kPart]: column sums by warp (16-byte rows, no bank conflicts)
  double *npart, *dpart;              // [kWarps]: squared norm of the next column, x^T A x
  double *d, *e, *tau, *V;
  int n, M, off;                         // basis size, frame rows, first used row of the frame
};

__device__ __forceinline__ constexpr int rblk(int I, int J) { return I * (I + 1) / 2 + J; }

// Sums 8 values over the 16 lanes of a half-warp; lane l ends with the total of value l >> 1.
__device__ __forceinline__ double sum16_of8(double (&v)[8], int lane) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double send = (lane & 8) ? v[k] : v[k + 4], keep = (lane & 8) ? v[k + 4] : v[k];
    v[k] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const double send = (lane & 4) ? v[k] : v[k + 2], keep = (lane & 4) ? v[k + 2] : v[k];
    v[k] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  }
  const double send = (lane & 2) ? v[0] : v[1], keep = (lane & 2) ? v[1] : v[0];
  const double r = keep + __shfl_xor_sync(0xffffffffu, send, 2);
  return r + __shfl_xor_sync(0xffffffffu, r, 1);
}
__device__ __forceinline__ double sum16_of2(double (&v)[2], int lane) {  // lane l: value l >> 3
  const double send = (lane & 8) ? v[0] : v[1], keep = (lane & 8) ? v[1] : v[0];
  double r = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  r += __shfl_xor_sync(0xffffffffu, r, 4);
  r += __shfl_xor_sync(0xffffffffu, r, 2);
  return r + __shfl_xor_sync(0xffffffffu, r, 1);
}
// The same for 4 values: lane l ends with the total of value l >> 2.
__device__ __forceinline__ double sum16_of4(double (&v)[4], int lane) {
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const double send = (lane & 8) ? v[k] : v[k + 2], keep = (lane & 8) ? v[k + 2] : v[k];
    v[k] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  const double send = (lane & 4) ? v[0] : v[1], keep = (lane & 4) ? v[1] : v[0];
  double r = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  r += __shfl_xor_sync(0xffffffffu, r, 2);
  return r + __shfl_xor_sync(0xffffffffu, r, 1);
}

// p[0] + ... + p[7], p 16-byte aligned
__device__ __forceinline__ double sum8(const double* p) {
  static_assert(kWarps == 8, "one term per warp");
  const double2* q = reinterpret_cast<const double2*>(p);
  const double2 a = q[0], b = q[1], c = q[2], d = q[3];
  return ((a.x + a.y) + (b.x + b.y)) + ((c.x + c.y) + (d.x + d.y));
}

// sqrt(x) and 1 / x for normal x > 0 by Newton-Raphson from the hardware's approximations (PTX rsqrt.approx.ftz.f64,
// rcp.approx.ftz.f64: by the PTX ISA formed from and given to 20 bits of the mantissa), without the branches of the library
// functions, so that the compiler can interleave the chain with the products around it. Two steps square an error of about 2^-19
// twice, below half an ulp; the root's residual x - y^2, exact by fma, then corrects the rounding of y = x r (2 ulp without).
// Against CUDA's sqrt and division: equal on 6e8 random values from 1e-240 to 1e239; the test holds 1 ulp.
__device__ __forceinline__ double sqrt_newton(double x) {
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
#pragma unroll
  for (int k = 0; k < 2; ++k) r = fma(0.5 * r, fma(-x * r, r, 1.0), r);
  const double y = x * r;
  return fma(0.5 * r, fma(-y, y, x), y);
}
__device__ __forceinline__ double rcp_newton(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
#pragma unroll
  for (int k = 0; k < 2; ++k) r = fma(r, fma(-x, r, 1.0), r);
  return r;
}

struct Refl {
  double beta, tau, v1;  // v1 = alpha - beta, the reflector's first element
};
// The reflector of the published column i: s = |x|^2, beta = -sign(alpha) |x|, tau = 2 / v^T v.
// A column below 1e-120 counts as reduced already (tau = 0).
__device__ __forceinline__ Refl reflector(const TriCtx& c, int i) {
  const double alpha = c.xs[i + 1], xn2 = sum8(c.npart), s = fma(alpha, alpha, xn2);
  const bool zero = !(xn2 > 1.0e-240);
  const double ss = zero ? 1.0 : s, nrm = sqrt_newton(ss);
  const double t = rcp_newton(fma(fabs(alpha), nrm, ss));
  Refl h;
  h.beta = zero ? alpha : -copysign(nrm, alpha);
  h.tau = zero ? 0.0 : t;
  h.v1 = alpha - h.beta;
  return h;
}

// Between the barriers of column i: thread t owns frame row p = first + t (rows below `first` are done).
// Completes y = A v, forms w = tau y + a2 v, and publishes v, w and the updated next column.
__device__ __forceinline__ void tri_rows(const TriCtx& c, int first, int i, const Refl& h) {
  const int t = threadIdx.x, p = first + t;
  double part = 0.0;
  if (p < c.M) {
    const double z1 = c.rsum[i + 1] + sum8(c.cpart + (i + 1) * kPart), raw1 = c.raw[i + 1];
    const double z = c.rsum[p] + sum8(c.cpart + p * kPart), raw = c.raw[p], x0 = c.xs[p];
    const double q = sum8(c.dpart);
    const double y1 = fma(-h.beta, raw1, z1), y = fma(-h.beta, raw, z);
    const double vav = fma(-h.beta, z1 + y1, q);  // x^T A x - 2 beta (A x)_{i+1} + beta^2 A_{i+1,i+1}
    const double a2 = -0.5 * h.tau * h.tau * vav;
    const double v = p == i + 1 ? h.v1 : x0;      // x is zero up to i
    const double w = p > i ? fma(h.tau, y, a2 * v) : 0.0;
    const double w1 = fma(h.tau, y1, a2 * h.v1);
    const double x = raw - fma(v, w1, w * h.v1);
    const double xn = p > i + 1 ? x : 0.0;
    c.xs[p] = xn;
    c.ws[p] = w;
    c.vs[p] = v;
    if (p > i + 2) part = x * x;
    if (p == i + 1) {
      c.d[p - c.off] = x;
      c.e[i - c.off] = h.beta;
      c.tau[i - c.off] = h.tau;
    }
  }
  if (first + (t & ~31) < c.M) part = warp_sum(part);
  if ((t & 31) == 0) c.npart[t >> 5] = part;
}

// After the second barrier: reflector i to global memory.
__device__ __forceinline__ void store_reflector(const TriCtx& c, int first, int i) {
  const int p = first + threadIdx.x;
  if (p > i && p < c.M) c.V[(i - c.off) * c.n + (p - c.off)] = c.vs[p];
}

// Columns of block column kRegB - NB of the register frame (frame rows base + 16 (kRegB - NB) ..),
// from frame row i on; returns the first column not done.
template <int NB>
__device__ __forceinline__ int tri_cols(double (&a)[kRegB * (kRegB + 1) / 2], const TriCtx& c, int base, int i) {
  constexpr int B0 = kRegB - NB;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, lane = tid & 31;
  const int end = min(base + 16 * (B0 + 1), c.M - 2);
  for (; i < end; ++i) {
    const Refl h = reflector(c, i);
    {
      double vc[NB], pc[NB], dot = 0.0;
#pragma unroll
      for (int k = 0; k < NB; ++k) {
        vc[k] = c.xs[base + 16 * (B0 + k) + tx];
        pc[k] = 0.0;
      }
      // the next column's present values
      if (tx == ((i + 1) & 15)) {
        const bool nextb = tx == 0;
#pragma unroll
        for (int I = 0; I < NB; ++I) {
          double x = a[rblk(B0 + I, B0)];
          if (I > 0) x = nextb ? a[rblk(B0 + I, B0 + (I > 0 ? 1 : 0))] : x;
          c.raw[base + 16 * (B0 + I) + ty] = x;
        }
      }
      // rows four blocks at a time: their sums over the 16 lanes of a row, and with the last ones x^T A x
#pragma unroll
      for (int I0 = 0; I0 < NB; I0 += 4) {
        constexpr bool kFull = (NB & 3) == 0;  // no free place beside the last rows
        double py[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int I = I0 + k;
          double acc = 0.0;
          if (I < NB) {
            const double vr = c.xs[base + 16 * (B0 + I) + ty];
#pragma unroll
            for (int J = 0; J <= I; ++J) {
              const double x = a[rblk(B0 + I, B0 + J)];
              acc = fma(x, vc[J], acc);
              if (J < I) pc[J] = fma(x, vr, pc[J]);
            }
            dot = fma(acc, vr, dot);
          }
          py[k] = acc;
        }
        const bool last = I0 + 4 >= NB;
        if (last) {
#pragma unroll
          for (int J = 0; J < NB; ++J) dot = fma(pc[J], vc[J], dot);
          if (!kFull) py[3] = dot;
        }
        const double sum = sum16_of4(py, lane);
        const int I = I0 + ((lane & 15) >> 2);
        if ((lane & 3) == 0 && I < NB) c.rsum[base + 16 * (B0 + I) + ty] = sum;
        if (last) {
          double q = sum;  // lane 12 of each half
          if (kFull) {
            q = dot;
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
          }
          q += __shfl_xor_sync(0xffffffffu, q, 16);
          if (lane == 12) c.dpart[tid >> 5] = q;
        }
      }
      // column sums over this warp's two rows of threads, then one partial per warp
#pragma unroll
      for (int J = 0; J < NB; ++J) pc[J] += __shfl_xor_sync(0xffffffffu, pc[J], 16);
      if (lane < 16) {
#pragma unroll
        for (int J = 0; J < NB; ++J) c.cpart[(base + 16 * (B0 + J) + tx) * kPart + (tid >> 5)] = pc[J];
      }
    }
    __syncthreads();
    tri_rows(c, base + 16 * B0, i, h);
    __syncthreads();
    store_reflector(c, base + 16 * B0, i);
    {
      double wr[NB], vr[NB];
#pragma unroll
      for (int I = 0; I < NB; ++I) {
        wr[I] = c.ws[base + 16 * (B0 + I) + ty];
        vr[I] = c.vs[base + 16 * (B0 + I) + ty];
      }
#pragma unroll
      for (int J = 0; J < NB; ++J) {
        const double wc = c.ws[base + 16 * (B0 + J) + tx], vc = c.vs[base + 16 * (B0 + J) + tx];
#pragma unroll
        for (int I = J; I < NB; ++I) {
          double& x = a[rblk(B0 + I, B0 + J)];
          x = fma(-wr[I], vc, fma(-vr[I], wc, x));
        }
      }
    }
  }
  return i;
}

// Private slot of this thread for block (I, J) of the memory columns (later columns, which live
// longer, come first and so stay in shared memory longest).
struct TriMem {
  double *sm, *gm;
  int cap, nbt, mb;  // slots in shared memory, blocks per frame side, memory block columns
  __device__ __forceinline__ double* at(int I, int J) const {
    // columns J+1 .. mb-1 hold nbt - J' blocks each
    const int k = mb - 1 - J;
    const int idx = k * (nbt - mb) + k * (k + 1) / 2, end = idx + nbt - J;  // a column is in one of the two
    return (end <= cap ? sm : gm) + (size_t)(idx + I - J) * kThreads + threadIdx.x;
  }
  __device__ __forceinline__ double* next(double* q) const { return q + kThreads; }  // the block below
};

// The columns of the memory block columns (n > kRegRows): the register blocks take part in every step.
__device__ __forceinline__ int tri_mem_cols(double (&a)[kRegB * (kRegB + 1) / 2], const TriCtx& c, const TriMem& m, int i) {
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, lane = tid & 31;
  const int mb = m.mb, base = 16 * mb;
  for (; i < base; ++i) {
    const int B = i >> 4;
    const Refl h = reflector(c, i);
    double py[8];
    double dot = 0.0;
    {
      double vc[kRegB], pc[kRegB];
#pragma unroll
      for (int k = 0; k < kRegB; ++k) {
        vc[k] = c.xs[base + 16 * k + tx];
        pc[k] = 0.0;
      }
#pragma unroll
      for (int I = 0; I < kRegB; ++I) {
        const double vr = c.xs[base + 16 * I + ty];
        double acc = 0.0;
#pragma unroll
        for (int J = 0; J <= I; ++J) {
          const double x = a[rblk(I, J)];
          acc = fma(x, vc[J], acc);
          if (J < I) pc[J] = fma(x, vr, pc[J]);
        }
        py[I] = acc;
      }
#pragma unroll
      for (int J = 0; J < kRegB; ++J) {
        dot = fma(pc[J], vc[J], dot);
        pc[J] += __shfl_xor_sync(0xffffffffu, pc[J], 16);
      }
      if (lane < 16) {
#pragma unroll
        for (int J = 0; J < kRegB; ++J) c.cpart[(base + 16 * J + tx) * kPart + (tid >> 5)] = pc[J];
      }
    }
    for (int J = B; J < mb; ++J) {
      const double vcj = c.xs[16 * J + tx];
      double pcj = 0.0;
      for (int I = J + 1; I < mb; ++I) pcj = fma(*m.at(I, J), c.xs[16 * I + ty], pcj);
      const double* q = m.at(mb, J);
#pragma unroll
      for (int k = 0; k < kRegB; ++k, q += kThreads) {
        const double x = *q;
        py[k] = fma(x, vcj, py[k]);
        pcj = fma(x, c.xs[base + 16 * k + ty], pcj);
      }
      dot = fma(pcj, vcj, dot);
      const double s = pcj + __shfl_xor_sync(0xffffffffu, pcj, 16);
      if (lane < 16) c.cpart[(16 * J + tx) * kPart + (tid >> 5)] = s;
    }
    for (int I = B; I < mb; ++I) {
      double acc = 0.0;
      for (int J = B; J <= I; ++J) acc = fma(*m.at(I, J), c.xs[16 * J + tx], acc);
      dot = fma(acc, c.xs[16 * I + ty], dot);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if ((lane & 15) == 0) c.rsum[16 * I + ty] = acc;
    }
#pragma unroll
    for (int I = 0; I < kRegB; ++I) dot = fma(py[I], c.xs[base + 16 * I + ty], dot);
    py[7] = dot;
    {
      const double s = sum16_of8(py, lane);
      const int I = (lane & 15) >> 1;
      const double both = s + __shfl_xor_sync(0xffffffffu, s, 16);
      if (!(lane & 1)) {
        if (I < kRegB) c.rsum[base + 16 * I + ty] = s;
        else if (lane < 16) c.dpart[tid >> 5] = both;
      }
    }
    if (tx == ((i + 1) & 15)) {
      const int Bn = (i + 1) >> 4;
      if (Bn < mb) {
        for (int I = Bn; I < m.nbt; ++I) c.raw[16 * I + ty] = *m.at(I, Bn);
      } else {
#pragma unroll
        for (int I = 0; I < kRegB; ++I) c.raw[base + 16 * I + ty] = a[rblk(I, 0)];
      }
    }
    __syncthreads();
    tri_rows(c, 16 * B, i, h);
    __syncthreads();
    store_reflector(c, 16 * B, i);
    double wr[kRegB], vr[kRegB];
#pragma unroll
    for (int k = 0; k < kRegB; ++k) {
      wr[k] = c.ws[base + 16 * k + ty];
      vr[k] = c.vs[base + 16 * k + ty];
    }
#pragma unroll
    for (int J = 0; J < kRegB; ++J) {
      const double wcj = c.ws[base + 16 * J + tx], vcj = c.vs[base + 16 * J + tx];
#pragma unroll
      for (int I = J; I < kRegB; ++I) a[rblk(I, J)] = fma(-wr[I], vcj, fma(-vr[I], wcj, a[rblk(I, J)]));
    }
    for (int J = B; J < mb; ++J) {
      const double vcj = c.vs[16 * J + tx], wcj = c.ws[16 * J + tx];
      for (int I = J; I < mb; ++I) {
        double* q = m.at(I, J);
        *q = fma(-c.ws[16 * I + ty], vcj, fma(-c.vs[16 * I + ty], wcj, *q));
      }
      double* q = m.at(mb, J);
#pragma unroll
      for (int k = 0; k < kRegB; ++k, q = m.next(q)) *q = fma(-wr[k], vcj, fma(-vr[k], wcj, *q));
    }
  }
  return i;
}

// The symmetric matrix to diagonalise: X, or (len > 0) sum_l coef[l] H_l over the accelerator's history
// matrices H_l = hist + ((head + l) % depth) stride; plus shift (I - proj). Lower triangles are read.
struct SymInput {
  const double* X;
  const double* hist;
  const double* coef;
  int head, len, depth;
  size_t stride;
  const double* proj;
  double shift;
};

// Householder reduction of the n x n symmetric matrix: diagonals to s.d, s.e,
// reflector scales to s.tau, reflector i to V[i n + r] (r > i).
// `gmem` holds the memory blocks that do not fit shared memory.
__device__ __noinline__ void tridiagonalize(int n, const SymInput& in, double* V, double* gmem, const EigenScratch& s) {
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  TriCtx c;
  c.n = n;
  c.M = frame_rows(n);
  c.off = c.M - n;
  c.xs = in_shared(s.sh);
  c.vs = c.xs + c.M;
  c.ws = c.vs + c.M;
  c.raw = c.ws + c.M;
  c.rsum = c.raw + c.M;
  c.cpart = c.rsum + c.M;  // M is even and sh 16-byte aligned: rows of kPart stay aligned
  c.npart = in_shared(s.red);
  c.dpart = c.npart + kWarps;
  c.d = in_shared(s.d);
  c.e = in_shared(s.e);
  c.tau = in_shared(s.tau);
  c.V = V;
  const int off = c.off, M = c.M, nbt = M / 16, mb = nbt - kRegB, base = 16 * mb;
  TriMem m;
  m.sm = s.sh + 15 * M;
  m.gm = gmem;
  m.cap = max(0, (s.sh_doubles - 15 * M) / kThreads);
  m.nbt = nbt;
  m.mb = mb;
  // Elements of the blocks at this thread, as indices into the lower triangle: affine in the block's coordinates, with other
  // constants on the diagonal (where both triangles are held). Negative columns are padding.
  const int r0 = ty - off, q0 = tx - off, hi0 = max(r0, q0), lo0 = min(r0, q0);
  auto col = [&](int I, int J) { return 16 * J + (I == J ? lo0 : q0); };
  auto index = [&](int I, int J) { return (16 * I + (I == J ? hi0 : r0)) * n + col(I, J); };
  const int terms = max(in.len, 1);
  auto source = [&](int l) { return in.len ? in.hist + (size_t)((in.head + l) % in.depth) * in.stride : in.X; };
  auto factor = [&](int l) { return in.len ? in.coef[l] : 1.0; };
  auto shifted = [&](int I, int J) { return in.shift * ((I == J && tx == ty ? 1.0 : 0.0) - in.proj[index(I, J)]); };
  // the memory blocks, 14 at a time: all their loads of one history matrix in flight together
  for (int J = 0; J < mb; ++J)
    for (int I0 = J; I0 < nbt; I0 += 14) {
      double x[14];
#pragma unroll
      for (int k = 0; k < 14; ++k) x[k] = 0.0;
      for (int l = 0; l < terms; ++l) {
        const double* __restrict__ src = source(l);
        const double cf = factor(l);
#pragma unroll
        for (int k = 0; k < 14; ++k)
          if (I0 + k < nbt && col(I0 + k, J) >= 0) x[k] = fma(cf, src[index(I0 + k, J)], x[k]);
      }
#pragma unroll
      for (int k = 0; k < 14; ++k)
        if (I0 + k < nbt) {
          if (in.shift != 0.0 && col(I0 + k, J) >= 0) x[k] += shifted(I0 + k, J);
          *m.at(I0 + k, J) = x[k];
        }
    }
  double a[kRegB * (kRegB + 1) / 2];
#pragma unroll
  for (int k = 0; k < kRegB * (kRegB + 1) / 2; ++k) a[k] = 0.0;
  // The register blocks from block F on: history matrices in groups of U, with all the group's loads in flight.
  auto load = [&](auto first, auto group) {
    constexpr int F = decltype(first)::value, U = decltype(group)::value;
    for (int l0 = 0; l0 < terms; l0 += U) {
      const double* src[U];
      double cf[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int l = min(l0 + u, terms - 1);
        src[u] = source(l);
        cf[u] = l0 + u >= terms ? 0.0 : factor(l);
      }
#pragma unroll
      for (int I = F; I < kRegB; ++I)
#pragma unroll
        for (int J = F; J <= I; ++J)
          if (col(mb + I, mb + J) >= 0) {
            const int ix = index(mb + I, mb + J);
            double x[U];
#pragma unroll
            for (int u = 0; u < U; ++u) x[u] = src[u][ix];
#pragma unroll
            for (int u = 0; u < U; ++u) a[rblk(I, J)] = fma(cf[u], x[u], a[rblk(I, J)]);
          }
    }
  };
  if (off >= 16 * (kRegB - 3)) load(std::integral_constant<int, kRegB - 3>{}, std::integral_constant<int, 4>{});
  else if (off >= 16 * (kRegB - 5)) load(std::integral_constant<int, kRegB - 5>{}, std::integral_constant<int, 2>{});
  else load(std::integral_constant<int, 0>{}, std::integral_constant<int, 1>{});
  if (in.shift != 0.0) {
#pragma unroll
    for (int I = 0; I < kRegB; ++I)
#pragma unroll
      for (int J = 0; J <= I; ++J)
        if (col(mb + I, mb + J) >= 0) a[rblk(I, J)] += shifted(mb + I, mb + J);
  }
  // publish the first column
  const int B = off >> 4;
  if (tx == (off & 15)) {
    if (B < mb) {
      for (int I = B; I < nbt; ++I) c.raw[16 * I + ty] = *m.at(I, B);
    } else {
#pragma unroll
      for (int J = 0; J < kRegB; ++J)
        if (J == B - mb) {
#pragma unroll
          for (int I = J; I < kRegB; ++I) c.raw[base + 16 * I + ty] = a[rblk(I, J)];
        }
    }
  }
  __syncthreads();
  double part = 0.0;
  if (tid < M) {
    const double x = tid > off ? c.raw[tid] : 0.0;
    c.xs[tid] = x;
    if (tid == off) c.d[0] = c.raw[tid];
    if (tid > off + 1) part = x * x;
  }
  part = warp_sum(part);
  if ((tid & 31) == 0) c.npart[tid >> 5] = part;
  __syncthreads();
  int i = off;
  if (mb > 0) i = tri_mem_cols(a, c, m, i);
  switch (mb > 0 ? kRegB : kRegB - (off >> 4)) {
    case 7: i = tri_cols<7>(a, c, base, i); [[fallthrough]];
    case 6: i = tri_cols<6>(a, c, base, i); [[fallthrough]];
    case 5: i = tri_cols<5>(a, c, base, i); [[fallthrough]];
    case 4: i = tri_cols<4>(a, c, base, i); [[fallthrough]];
    case 3: i = tri_cols<3>(a, c, base, i); [[fallthrough]];
    case 2: i = tri_cols<2>(a, c, base, i); [[fallthrough]];
    default: tri_cols<1>(a, c, base, i);
  }
  if (tid == 0) {
    if (n >= 2) {
      c.e[n - 2] = c.xs[M - 1];
      c.tau[n - 2] = 0.0;
    }
    c.e[n - 1] = 0.0;
  }
  if (n >= 2 && tid == kThreads - 1) c.d[n - 1] = a[rblk(kRegB - 1, kRegB - 1)];
  __syncthreads();
}

// ------------------------------------------------------------- 2. split + eigenvalues
// Sturm count: number of eigenvalues of T[lo..hi] below x.
__device__ __forceinline__ int sturm(const double* d, const double* e2, int lo, int hi, double x, double pivmin) {
  int cnt = 0;
  double q = d[lo] - x;
  if (fabs(q) < pivmin) q = -pivmin;
  cnt += q < 0.0;
  for (int i = lo + 1; i <= hi; ++i) {
    q = (d[i] - x) - e2[i - 1] / q;
    if (fabs(q) < pivmin) q = -pivmin;
    cnt += q < 0.0;
  }
  return cnt;
}

// Power of two that brings the larger of two magnitudes into [1, 2), as its exponent (0 for zeros).
__device__ __forceinline__ int pair_exponent(double a, double b) {
  const double m = fmax(fabs(a), fabs(b));
  const int ex = (__double2hiint(m) >> 20) & 0x7ff;
  return ex == 0 ? 0 : ex - 1023;
}
// A number that orders the magnitudes p 2^ex (p >= 0): exponent plus fraction, a piecewise linear log2.
__device__ __forceinline__ double scaled_order(double p, int ex) {
  const int hi = __double2hiint(p), e = hi >> 20;
  if (e == 0) return -INFINITY;
  return (double)(e + ex) + (__hiloint2double((hi & 0xfffff) | 0x3ff00000, __double2loint(p)) - 1.0);
}
__device__ __forceinline__ double pow2(int ex) {  // 2^ex for normal results, 0 below, the largest power above
  return ex < -1022 ? 0.0 : __hiloint2double((min(ex, 1023) + 1023) << 20, 0);
}

// Sturm counts at M shifts at once, without divisions (see the ratio form above for the
// reference recurrence): p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2}; sign changes between
// consecutive values count the eigenvalues below x. Pairs are rescaled by powers of two every
// 8 steps (each step grows |p| by far less than 2^32 for the matrices here), exact for ratios.
// val[t] 2^(256 ex[t]) is the characteristic polynomial at x[t].
template <int M>
__device__ __forceinline__ void sturm_multi(const double* __restrict__ d, const double* __restrict__ e2, int n,
                                            const double (&x)[M], int (&cnt)[M], double (&val)[M], int (&ex)[M]) {
  constexpr int kOne = 1023 << 20, kBig = (1023 + 256) << 20, kSmall = (1023 - 256) << 20;  // upper halves of 1, 2^256, 2^-256
  double p[M], pm[M];
  unsigned sg[M];  // sign bits, the newest last
#pragma unroll
  for (int t = 0; t < M; ++t) {
    pm[t] = 1.0;
    ex[t] = 0;
    p[t] = d[0] - x[t];
    sg[t] = (unsigned)__double2hiint(p[t]) >> 31;
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
        sg[t] = __funnelshift_l((unsigned)__double2hiint(pn), sg[t], 1);
        pm[t] = p[t];
        p[t] = pn;
      }
    }
#pragma unroll
    for (int t = 0; t < M; ++t) {
      cnt[t] += __popc((sg[t] ^ (sg[t] >> 1)) & 0xffu);
      const int m = max(__double2hiint(p[t]) & 0x7fffffff, __double2hiint(pm[t]) & 0x7fffffff);  // the larger magnitude's upper half
      const int up = m > kBig ? 1 : (m < kSmall ? -1 : 0);
      const double sc = __hiloint2double(kOne - up * (256 << 20), 0);
      ex[t] += up;
      p[t] *= sc;
      pm[t] *= sc;
    }
  }
  const unsigned left = (1u << (n - i)) - 1u;
  for (; i < n; ++i) {
    const double di = d[i], ei = e2[i - 1];
#pragma unroll
    for (int t = 0; t < M; ++t) {
      const double pn = fma(di - x[t], p[t], -ei * pm[t]);
      sg[t] = __funnelshift_l((unsigned)__double2hiint(pn), sg[t], 1);
      pm[t] = p[t];
      p[t] = pn;
    }
  }
#pragma unroll
  for (int t = 0; t < M; ++t) cnt[t] += __popc((sg[t] ^ (sg[t] >> 1)) & left);
#pragma unroll
  for (int t = 0; t < M; ++t) val[t] = p[t];
}

// Eigenvalue j of T by multisection: a group of g lanes (a power of two, at most 32) brackets it; each step the group takes Sturm counts at P = g * kPts points (kPts
// per lane, evaluated together) and keeps the interval between the neighbouring two that holds it.
// Invariant: count(lo) <= j < count(hi). The points are evenly spaced (the bracket shrinks by P + 1) until
// the interval holds this eigenvalue alone. From then on they close in geometrically on the
// secant estimate of the characteristic polynomial's root, whose values the counts yield on the way; the counts
// still decide, and a step that gained less than a factor of 4 is followed by an even one. The search ends at an interval of
// 2 eps |lambda|, whatever the norm.
// What bounds it: the recurrence, about 40 cycles a row and step; steps from a cold start at n = 64, k = 33:
// 17 when all were even, 9 now.
// With `prev` (eigenvalue j of the previous SCF iteration) and `dprev` (its last change) the search starts from a
// bracket around prev[j] once two counts confirm it. Whole warps call; lanes without an eigenvalue pass
// active = false.
__device__ __forceinline__ double multisect(const double* __restrict__ d, const double* __restrict__ e2, int n, int j,
                                            bool active, int g, double glo, double ghi, double pivmin, double tnorm,
                                            const double* prev, const double* dprev) {
  constexpr double eps = 2.220446049250313e-16;
  constexpr int kPts = 2;
  const int P = g * kPts;
  const int lane = threadIdx.x & 31;
  const int gbase = lane & ~(g - 1), gl = lane & (g - 1);
  const unsigned gbits = g == 32 ? 0xffffffffu : ((1u << g) - 1u);
  double lo = glo, hi = ghi;
  double flo = 0.0, fhi = 0.0;  // polynomial at lo and hi, 0 while unknown
  int elo = 0, ehi = 0, clo = 0, chi = n;
  if (prev) {
    // warm bracket around the previous SCF iteration's value, widened until two Sturm
    // counts confirm that it holds eigenvalue j (else the Gershgorin interval stays)
    const double c0 = active ? prev[j] : 0.0;
    const double w0 = active ? fmax(4.0 * fabs(dprev[j]), 1.0e-9 * fmax(tnorm, 1.0)) : 0.0;
    double x[4], fv[4];
    int cn[4], fe[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {  // brackets w0 and 64 w0: lower ends on even t, upper on odd
      const double w = w0 * (t >= 2 ? 64.0 : 1.0);
      x[t] = (t & 1) ? fmin(c0 + w, ghi) : fmax(c0 - w, glo);
    }
    if (active) sturm_multi<4>(d, e2, n, x, cn, fv, fe);
    if (active) {
#pragma unroll
      for (int t = 2; t >= 0; t -= 2)  // the narrow one last
        if (x[t] < x[t + 1] && cn[t] <= j && cn[t + 1] >= j + 1) {
          lo = x[t];
          hi = x[t + 1];
          flo = fv[t];
          fhi = fv[t + 1];
          elo = fe[t];
          ehi = fe[t + 1];
          clo = cn[t];
          chi = cn[t + 1];
        }
    }
  }
  bool act = active, even = false;
  for (int it = 0; it < 160; ++it) {
    if (act) {
      const double mid = 0.5 * (lo + hi);
      if (hi - lo <= 2.0 * eps * fmax(fabs(lo), fabs(hi)) + 4.0 * pivmin || !(mid > lo && mid < hi)) act = false;
    }
    if (!__any_sync(0xffffffffu, act)) break;
    const double w = hi - lo;
    const bool close = !even && clo == j && chi == j + 1 && flo != 0.0 && fhi != 0.0;
    double x[kPts], fv[kPts];
    int cn[kPts], fe[kPts];
    if (close) {
      const double a = fabs(flo), b = fabs(fhi);  // the one of the smaller scale counts as 0
      const double r = elo == ehi ? a / (a + b) : (elo > ehi ? 1.0 : 0.0);
      const double xs = lo + w * r, tiny = eps * fmax(fabs(lo), fabs(hi));
#pragma unroll
      for (int t = 0; t < kPts; ++t) {  // distances w/4 .. w/2^26 (w/16 for P = 2), below and above
        const int q = gl * kPts + t, k = q < g ? q : P - 1 - q;
        const int ex = g == 1 ? 4 : 2 + 24 * k / (g - 1);
        const double dl = fmax(w * pow2(-ex), tiny);
        x[t] = fmin(fmax(q < g ? xs - dl : xs + dl, lo), hi);
      }
    } else {
#pragma unroll
      for (int t = 0; t < kPts; ++t) x[t] = lo + w * (double)(gl * kPts + t + 1) / (double)(P + 1);
    }
    if (act) sturm_multi<kPts>(d, e2, n, x, cn, fv, fe);
    int tf = kPts;  // this lane's first point above eigenvalue j
#pragma unroll
    for (int t = kPts - 1; t >= 0; --t)
      if (act && cn[t] > j) tf = t;
    const unsigned bal = __ballot_sync(0xffffffffu, act && tf < kPts);
    const unsigned mine = (bal >> gbase) & gbits;
    // upper end: point f (the first above), lower end: point f - 1; either may be the bracket's own end
    const int hl = mine ? gbase + __ffs(mine) - 1 : gbase + g - 1;
    const int th = __shfl_sync(0xffffffffu, tf, hl);
    const int f = mine ? (hl - gbase) * kPts + th : P;
    auto take = [&](int q, double& px, double& pf, int& pe, int& pc) {  // point q of the group (any lane asks)
      const int src = gbase + min(max(q, 0), P - 1) / kPts, tt = min(max(q, 0), P - 1) % kPts;
      double vx = 0.0, vf = 0.0;
      int ve = 0, vc = 0;
#pragma unroll
      for (int t = 0; t < kPts; ++t) {
        const double sx = __shfl_sync(0xffffffffu, x[t], src), sf = __shfl_sync(0xffffffffu, fv[t], src);
        const int se = __shfl_sync(0xffffffffu, fe[t], src), sc = __shfl_sync(0xffffffffu, cn[t], src);
        if (t == tt) {
          vx = sx;
          vf = sf;
          ve = se;
          vc = sc;
        }
      }
      if (q >= 0 && q < P && act) {
        px = vx;
        pf = vf;
        pe = ve;
        pc = vc;
      }
    };
    double nlo = lo, nhi = hi;
    take(f - 1, nlo, flo, elo, clo);
    take(f, nhi, fhi, ehi, chi);
    if (act) {
      if (!(nhi - nlo < w)) {
        if (close) even = true;  // no gain around the estimate: split evenly
        else act = false;
      } else {
        even = close && (nhi - nlo) * 4.0 > w;
        lo = nlo;
        hi = nhi;
      }
    }
  }
  return 0.5 * (lo + hi);
}

// Splits T where the coupling is negligible and computes the lowest `kval` eigenvalues.
// Leaves pivmin / tnorm in misc[0] / misc[1]. With `prev` (the same eigenvalues of the
// previous SCF iteration) and `dprev` (their last change) the search starts from a bracket
// around prev[j] once Sturm counts confirm it.
__device__ void tridiag_eigenvalues(int n, int kval, const EigenScratch& s_, const double* prev = nullptr,
                                    const double* dprev = nullptr) {
  struct {
    double *d, *e, *e2, *misc, *lam;
    int *blk, *nblk;
  } s = {in_shared(s_.d), in_shared(s_.e), in_shared(s_.e2), in_shared(s_.misc), in_shared(s_.lam), in_shared(s_.blk),
         in_shared(s_.nblk)};
  const int tid = threadIdx.x;
  constexpr double eps = 2.220446049250313e-16;
  {
    // Gershgorin bounds of the unsplit T, then split where |e_i| <= 1000 eps ||T||: an
    // absolute criterion, so exactly degenerate eigenvalues (which Householder leaves joined
    // by couplings of a few eps ||T||) land in separate blocks. One row per thread (n <= kThreads).
    const bool row = tid < n;
    const double ei = tid + 1 < n ? s.e[tid] : 0.0;
    const double rad = fabs(ei) + (row && tid > 0 ? fabs(s.e[tid - 1]) : 0.0);
    const double gl = -block_max(row ? rad - s.d[tid] : -INFINITY, s_.red);
    const double gu = block_max(row ? s.d[tid] + rad : -INFINITY, s_.red);
    const double tnorm = fmax(fabs(gl), fabs(gu));
    const bool cut = tid + 1 < n && fabs(ei) <= 1000.0 * eps * tnorm;
    if (row) s.e2[tid] = cut ? 0.0 : ei * ei;
    const double emax = block_max(row && !cut ? ei * ei : 0.0, s_.red);
    if (cut) s.e[tid] = 0.0;
    if (__syncthreads_or(cut)) {
      if (tid == 0) {
        int nb = 0;
        s.blk[0] = 0;
        for (int i = 0; i + 1 < n; ++i)
          if (s.e[i] == 0.0) s.blk[++nb] = i + 1;
        s.blk[++nb] = n;
        *s.nblk = nb;
      }
    } else if (tid == 0) {
      s.blk[0] = 0;
      s.blk[1] = n;
      *s.nblk = 1;
    }
    if (tid == 0) {
      s.misc[0] = 2.2250738585072014e-308 * fmax(1.0, emax);  // pivmin
      s.misc[1] = tnorm;
      s.misc[2] = gl - 4.0 * eps * tnorm * n - 1.0e-300;
      s.misc[3] = gu + 4.0 * eps * tnorm * n + 1.0e-300;
    }
  }
  __syncthreads();
  const double pivmin = s.misc[0], tnorm = s.misc[1], glo = s.misc[2], ghi = s.misc[3];
  // a group of g lanes per eigenvalue (a power of two, g <= 32, kval * g <= kThreads)
  int g = 1;
  while (g < 32 && kval * (2 * g) <= kThreads) g *= 2;
  for (int j0 = 0; j0 < kval; j0 += kThreads / g) {
    const int j = j0 + tid / g;
    const double v = multisect(s.d, s.e2, n, j, j < kval, g, glo, ghi, pivmin, tnorm, prev, dprev);
    if (j < kval && (tid & (g - 1)) == 0) s.lam[j] = v;
  }
  __syncthreads();
}

// ------------------------------------------------------------- 3. tridiagonal eigenvectors
// Eigenvectors j < kvec of T, unnormalised, into Yt[i kvec + j] (zero outside the block of each). `tf` is
// per-CTA global scratch of 6 n^2 doubles. Every array has the vector index fastest, so that the
// threads of a warp (one vector each) touch consecutive addresses.
//
// The twisted factorisation N_r D_r N_r^T of T - lam gives y from the top down to row r and from the bottom up to it.
// Both parts obey T's own three-term recurrence: f_{i+1} = ((lam - d_i) f_i - e_{i-1} f_{i-1}) / e_i
// from f = 1 in the first row, and g likewise upward from the last row. One half of the CTA runs f, the other
// g; with the reciprocals of e shared by all vectors, one FMA a row is in the dependent chain (the
// pivots L+ D+ L+^T, U- D- U-^T of the same factorisation have a division in it: 150 cycles a row).
// The twist gamma_r is 1 / [(T - lam)^-1]_rr up to a factor common to all rows, and that element is
// proportional to f_r g_r, so r is the row of the largest |f g|; y = f / f_r above it, g / g_r below.
// Pairs are rescaled by powers of two every 8 rows (a row grows them by at most (lam - d) / e, and e
// is above 1000 eps ||T|| within a block); the exponents are kept per group of 8 rows.
__device__ double* tridiag_vectors(int n, int kvec, double* tf, const EigenScratch& s_) {
  struct {
    const double *d, *e, *e2, *lam, *misc;
    const int *blk, *nblk;
    int* vinfo;
    double *inve, *aux;
  } s = {in_shared(s_.d),   in_shared(s_.e),    in_shared(s_.e2),    in_shared(s_.lam), in_shared(s_.misc),
         in_shared(s_.blk), in_shared(s_.nblk), in_shared(s_.vinfo), in_shared(s_.p),   in_shared(s_.v)};
  const int tid = threadIdx.x;
  const double pivmin = s.misc[0], tnorm = s.misc[1];
  const int nb = *s.nblk;
  const double win = 1.0e-11 * fmax(tnorm, 1.0);
  const size_t nk = (size_t)n * kvec;
  double* __restrict__ F = tf;
  double* __restrict__ G = tf + nk;
  double* __restrict__ Yt = tf + 2 * nk;
  int* __restrict__ EF = reinterpret_cast<int*>(tf + 3 * nk);  // [group of 8 block rows][kvec]
  int* __restrict__ EG = EF + (size_t)((n + 7) / 8) * kvec;
  constexpr int kHalf = kThreads / 2;
  const int half = tid / kHalf, hj = tid % kHalf;
  if (tid < n) s.inve[tid] = s.e[tid] != 0.0 ? 1.0 / s.e[tid] : 0.0;
  __syncthreads();
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
    const int lo = s.blk[b], m = s.blk[b + 1] - lo;
    // step t of half 0 goes from row lo + t to the next; of half 1 from row hi - t to the one before
    const int step = half == 0 ? 1 : -1;
    const double* dd = s.d + (half == 0 ? lo : lo + m - 1);
    const double* ee = s.e + (half == 0 ? lo : lo + m - 2);       // coupling crossed by step t
    const double* iv = s.inve + (half == 0 ? lo : lo + m - 2);
    double* __restrict__ out = (half == 0 ? F : G) + (size_t)(half == 0 ? lo : lo + m - 1) * kvec + j;
    int* __restrict__ ex = (half == 0 ? EF : EG) + j;
    const ptrdiff_t os = (ptrdiff_t)step * kvec;
    double f = 1.0, fm = 0.0;  // this row's value and the one before
    int e = 0;
    *out = f;
    *ex = 0;
    for (int t0 = 0; t0 < m - 1; t0 += 8) {
      double A[8], B[8], y[8];  // the eight rows' coefficients first: only FMAs stay in the chain
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int t = min(t0 + u, m - 2);
        const double inv = iv[step * t];
        A[u] = (lam - dd[step * t]) * inv;
        B[u] = t > 0 ? ee[step * (t - 1)] * inv : 0.0;
      }
      if (t0 > 0) {
        const int q = pair_exponent(f, fm);
        const double sc = pow2(-q);
        f *= sc;
        fm *= sc;
        e += q;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const double fn = fma(A[u], f, -(B[u] * fm));
        fm = f;
        f = y[u] = fn;
      }
      ex[(size_t)(t0 >> 3) * kvec] = e;  // of rows t0 + 1 .. t0 + 8 of the block
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (t0 + u < m - 1) out[os * (t0 + u + 1)] = y[u];
    }
  }
  __syncthreads();
  // From here every thread has one vector and a share of its groups of 8 rows (vectors fastest; more than 16
  // shares would only lengthen the combination).
  // Row lo + t of f is in group (t - 1) / 8 (row lo in group 0, whose exponent is 0), of g row hi - t.
  const int shares = min(kThreads / kvec, 16), share = tid / kvec, jv = tid - share * kvec;
  const bool in_share = share < shares;
  // The row of the largest |f g|.
  double* __restrict__ K = in_shared(s_.sh);                                       // [shares][kvec], at most kThreads
  int* __restrict__ R = reinterpret_cast<int*>(in_shared(s_.sh) + kThreads);       // the same
  if (in_share) {
    const int j = jv, b = s.vinfo[j], lo = s.blk[b], hi = s.blk[b + 1] - 1;
    double best = -INFINITY;
    int br = hi;
    for (int g = share; lo + 8 * g <= hi; g += shares) {
      const int t0 = 8 * g + (g > 0 ? 1 : 0), t1 = min(8 * g + 8, hi - lo);  // rows t0 .. t1 of the block
      const int ef = EF[g * kvec + j];
      // g's rows hi - i: nine consecutive rows meet at most two of its groups
      const int gb = max(hi - lo - t1 - 1, 0) >> 3;
      const int e0 = EG[gb * kvec + j], e1 = EG[min(gb + 1, (n + 7) / 8 - 1) * kvec + j];
      double p[9];
#pragma unroll
      for (int u = 0; u < 9; ++u) {
        const int i = lo + min(t0 + u, t1);
        p[u] = fabs(F[i * kvec + j] * G[i * kvec + j]);
      }
#pragma unroll
      for (int u = 0; u < 9; ++u) {
        const int t = t0 + u;
        if (t <= t1) {
          const double key = scaled_order(p[u], ef + ((max(hi - lo - t - 1, 0) >> 3) == gb ? e0 : e1));
          if (key > best) {
            best = key;
            br = lo + t;
          }
        }
      }
    }
    K[share * kvec + j] = best;
    R[share * kvec + j] = br;
  }
  __syncthreads();
  if (tid < kvec) {
    const int j = tid;
    double best = K[j];
    int r = R[j];
    for (int q = 1; q < shares; ++q)
      if (K[q * kvec + j] > best) {
        best = K[q * kvec + j];
        r = R[q * kvec + j];
      }
    const int b = s.vinfo[j], lo = s.blk[b];
    s.vinfo[j] = b | ((r - lo) << 16);
    s.inve[j] = 1.0 / F[r * kvec + j];  // the reciprocals of e are spent by now
    s.aux[j] = 1.0 / G[r * kvec + j];
  }
  __syncthreads();
  if (in_share) {
    const int j = jv, vi = s.vinfo[j], b = vi & 0xffff, lo = s.blk[b], hi = s.blk[b + 1] - 1, r = lo + (vi >> 16);
    const double rf = s.inve[j], rg = s.aux[j];
    const int ef = EF[(max(r - lo - 1, 0) >> 3) * kvec + j], eg = EG[(max(hi - r - 1, 0) >> 3) * kvec + j];
    for (int i0 = 8 * share; i0 < n; i0 += 8 * shares) {
      double y[8];
      int q[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int i = min(i0 + u, n - 1);
        const bool up = i < r;
        const bool in = i >= lo && i <= hi;
        const double* src = up ? F : G;
        const int* es = up ? EF : EG;
        const int t = up ? i - lo : hi - i;
        y[u] = in ? src[i * kvec + j] : 0.0;
        q[u] = in ? es[(max(t - 1, 0) >> 3) * kvec + j] : 0;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const bool up = i0 + u < r;
        if (i0 + u < n) Yt[(i0 + u) * kvec + j] = y[u] * (up ? rf : rg) * pow2(q[u] - (up ? ef : eg));
      }
    }
  }
  __syncthreads();
  // Eigenvalues of one block closer than 1e-7 ||T||: the twisted vectors are not reliable
  // there, so every cluster member after the first is recomputed by inverse iteration on a
  // row-pivoted LU of T_b - lam, re-orthogonalised against the earlier members of its
  // cluster (the dstein scheme). One thread per block; clusters are rare.
  const double ctol = 1.0e-7 * fmax(tnorm, 1.0), tiny = 2.220446049250313e-16 * fmax(tnorm, 1.0);
  const bool close = tid > 0 && tid < kvec && s.lam[tid] - s.lam[tid - 1] < ctol;  // kvec <= kThreads
  if (!__syncthreads_or(close || nb > 1)) return Yt;
  for (int b = tid; b < nb; b += kThreads) {
    const int lo = s.blk[b], hi = s.blk[b + 1] - 1, m = hi - lo + 1;
    int head = -1, prev = -1;
    for (int j = 0; j < kvec; ++j) {
      if ((s.vinfo[j] & 0xffff) != b) continue;
      if (prev < 0 || s.lam[j] - s.lam[prev] >= ctol) {
        head = j;
        prev = j;
        continue;
      }
      if (prev == head) {  // the cluster's first vector is orthogonalised against: normalise it
        double nrm = 0.0;
        for (int i = lo; i <= hi; ++i) nrm += Yt[(size_t)i * kvec + head] * Yt[(size_t)i * kvec + head];
        nrm = 1.0 / sqrt(nrm);
        for (int i = lo; i <= hi; ++i) Yt[(size_t)i * kvec + head] *= nrm;
      }
      prev = j;
      // the LU factors take this vector's columns of scratch that is spent by now
      auto dd = [&](int i) -> double& { return F[(size_t)(lo + i) * kvec + j]; };
      auto dl = [&](int i) -> double& { return G[(size_t)(lo + i) * kvec + j]; };
      auto du = [&](int i) -> double& { return tf[3 * nk + (size_t)(lo + i) * kvec + j]; };
      auto du2 = [&](int i) -> double& { return tf[4 * nk + (size_t)(lo + i) * kvec + j]; };
      unsigned pv[kMaxN / 32];
#pragma unroll
      for (int q = 0; q < kMaxN / 32; ++q) pv[q] = 0u;
      const double sg = s.lam[j];
      for (int i = 0; i < m; ++i) {
        dd(i) = s.d[lo + i] - sg;
        if (i + 1 < m) dl(i) = du(i) = s.e[lo + i];
      }
      for (int i = 0; i + 1 < m; ++i) {
        if (fabs(dd(i)) >= fabs(dl(i))) {
          if (dd(i) == 0.0) dd(i) = tiny;
          const double f = dl(i) / dd(i);
          dl(i) = f;
          dd(i + 1) -= f * du(i);
          if (i + 2 < m) du2(i) = 0.0;
        } else {
          const double f = dd(i) / dl(i);
          dd(i) = dl(i);
          dl(i) = f;
          const double t = du(i);
          du(i) = dd(i + 1);
          dd(i + 1) = t - f * dd(i + 1);
          if (i + 2 < m) {
            du2(i) = du(i + 1);
            du(i + 1) = -f * du(i + 1);
          }
          pv[i >> 5] |= 1u << (i & 31);
        }
      }
      for (int i = 0; i < m; ++i)
        if (fabs(dd(i)) < tiny) dd(i) = dd(i) < 0.0 ? -tiny : tiny;
      auto x = [&](int i) -> double& { return Yt[(size_t)(lo + i) * kvec + j]; };
      for (int i = 0; i < m; ++i) x(i) = sin(1.0 + 0.7 * i + 1.3 * j);
      for (int it = 0; it < 3; ++it) {
        for (int i = 0; i + 1 < m; ++i) {
          if (!((pv[i >> 5] >> (i & 31)) & 1u)) {
            x(i + 1) -= dl(i) * x(i);
          } else {
            const double t = x(i);
            x(i) = x(i + 1);
            x(i + 1) = t - dl(i) * x(i);
          }
        }
        x(m - 1) /= dd(m - 1);
        if (m > 1) x(m - 2) = (x(m - 2) - du(m - 2) * x(m - 1)) / dd(m - 2);
        for (int i = m - 3; i >= 0; --i) x(i) = (x(i) - du(i) * x(i + 1) - du2(i) * x(i + 2)) / dd(i);
        for (int pass = 0; pass < 2; ++pass)
          for (int q = head; q < j; ++q) {
            if ((s.vinfo[q] & 0xffff) != b) continue;
            double dot = 0.0;
            for (int i = 0; i < m; ++i) dot += Yt[(size_t)(lo + i) * kvec + q] * x(i);
            for (int i = 0; i < m; ++i) x(i) -= dot * Yt[(size_t)(lo + i) * kvec + q];
          }
        double nrm = 0.0;
        for (int i = 0; i < m; ++i) nrm += x(i) * x(i);
        nrm = 1.0 / sqrt(nrm);
        for (int i = 0; i < m; ++i) x(i) *= nrm;
      }
    }
  }
  __syncthreads();
  return Yt;
}

// ------------------------------------------------------------------- 4. back-transform
// Y[j] <- H(0) H(1) ... H(n-3) y_j for j < kvec. A group of G lanes holds NV vectors, RT rows of each
// per lane (n <= G RT). The reflectors pass through shared memory eight at a time (one warp
// copies one), double buffered with the next eight in registers; the NV dot products
// are summed over the group together. With at most 16 values of z a lane two reflectors are applied at a time, v0^T
// H1 z = v0^T z - tau1 (v1^T z) (v0^T v1), so one round of shuffles serves both (n = 48: 20.3k cycles one at a
// time, 17.6k in pairs; with more, two reflectors and z do not fit the registers: n = 128 95k against 129k). Half of the rows are skipped once they lie above the reflectors.
template <int G, int RT, int NV>
__device__ __forceinline__ void back_transform_t(int n, int kvec, const double* __restrict__ V,
                                                 const double* __restrict__ Yt, double* Y,
                                                 const double* __restrict__ tau_, double* sh) {
  constexpr int NG = kThreads / G, LD = G * RT, NP = (LD + 31) / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gl = tid % G, g = tid / G;
  const int c0 = n >= 3 ? (n - 3) / 8 : -1;
  for (int j0 = 0; j0 < kvec; j0 += NG * NV) {
    double z[NV][RT];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int j = j0 + v * NG + g;
#pragma unroll
      for (int t = 0; t < RT; ++t) {
        const int r = gl + G * t;
        z[v][t] = r < n && j < kvec ? Yt[(size_t)r * kvec + j] : 0.0;
      }
    }
    {  // unit norm
      double nv[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        double q0 = 0.0, q1 = 0.0;
#pragma unroll
        for (int t = 0; t < RT; t += 2) {
          q0 = fma(z[v][t], z[v][t], q0);
          if (t + 1 < RT) q1 = fma(z[v][t + 1], z[v][t + 1], q1);
        }
        nv[v] = q0 + q1;
      }
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
        for (int v = 0; v < NV; ++v) nv[v] += __shfl_xor_sync(0xffffffffu, nv[v], o);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        nv[v] = nv[v] > 0.0 ? 1.0 / sqrt(nv[v]) : 0.0;
#pragma unroll
        for (int t = 0; t < RT; ++t) z[v][t] *= nv[v];
      }
    }
    double nx[NP];
    auto fetch = [&](int c) {
      const int i = 8 * c + warp;
#pragma unroll
      for (int u = 0; u < NP; ++u) {
        const int r = lane + 32 * u;
        nx[u] = i <= n - 3 && r > i && r < n ? V[(size_t)i * n + r] : 0.0;
      }
    };
    // stages c0 .. c1 (descending); rows of lane index below T0 are above all their reflectors
    auto stages = [&](auto first, int cs, int ce) {
      constexpr int T0 = decltype(first)::value;
      for (int c = cs; c >= ce; --c) {
        double* buf = sh + (c & 1) * 8 * LD;
#pragma unroll
        for (int u = 0; u < NP; ++u)
          if (lane + 32 * u < LD) buf[warp * LD + lane + 32 * u] = nx[u];
        __syncthreads();
        if (c > 0) fetch(c - 1);
        if constexpr (RT * NV <= 16) {
#pragma unroll 1
          for (int u = 7; u > 0; u -= 2) {  // H(i + 1), then H(i)
            const int i = 8 * c + u - 1;
            if (i > n - 3) continue;
            const double t1 = i + 1 <= n - 3 ? tau_[i + 1] : 0.0, t0 = tau_[i];
            const double* __restrict__ w1 = buf + u * LD + gl;
            const double* __restrict__ w0 = w1 - LD;
            double a1[NV], a0[NV], gm = 0.0;
#pragma unroll
            for (int v = 0; v < NV; ++v) a1[v] = a0[v] = 0.0;
#pragma unroll
            for (int t = T0; t < RT; ++t) {
              const double p1 = w1[G * t], p0 = w0[G * t];
#pragma unroll
              for (int v = 0; v < NV; ++v) {
                a1[v] = fma(p1, z[v][t], a1[v]);
                a0[v] = fma(p0, z[v][t], a0[v]);
              }
              gm = fma(p1, p0, gm);
            }
#pragma unroll
            for (int o = G / 2; o > 0; o >>= 1) {
#pragma unroll
              for (int v = 0; v < NV; ++v) {
                a1[v] += __shfl_xor_sync(0xffffffffu, a1[v], o);
                a0[v] += __shfl_xor_sync(0xffffffffu, a0[v], o);
              }
              gm += __shfl_xor_sync(0xffffffffu, gm, o);
            }
#pragma unroll
            for (int v = 0; v < NV; ++v) {
              a1[v] *= -t1;
              a0[v] = -t0 * fma(a1[v], gm, a0[v]);
            }
#pragma unroll
            for (int t = T0; t < RT; ++t) {
              const double p1 = w1[G * t], p0 = w0[G * t];
#pragma unroll
              for (int v = 0; v < NV; ++v) z[v][t] = fma(a0[v], p0, fma(a1[v], p1, z[v][t]));
            }
          }
        } else {
#pragma unroll 1
          for (int u = 7; u >= 0; --u) {
            const int i = 8 * c + u;
            if (i > n - 3) continue;
            const double tau = tau_[i];
            const double* __restrict__ w = buf + u * LD + gl;
            double vr[RT], a0[NV], a1[NV];
#pragma unroll
            for (int t = T0; t < RT; ++t) vr[t] = w[G * t];
#pragma unroll
            for (int v = 0; v < NV; ++v) a0[v] = a1[v] = 0.0;
#pragma unroll
            for (int t = T0; t < RT; t += 2)
#pragma unroll
              for (int v = 0; v < NV; ++v) {
                a0[v] = fma(vr[t], z[v][t], a0[v]);
                if (t + 1 < RT) a1[v] = fma(vr[t + 1], z[v][t + 1], a1[v]);
              }
#pragma unroll
            for (int v = 0; v < NV; ++v) a0[v] += a1[v];
#pragma unroll
            for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
              for (int v = 0; v < NV; ++v) a0[v] += __shfl_xor_sync(0xffffffffu, a0[v], o);
#pragma unroll
            for (int v = 0; v < NV; ++v) a0[v] *= -tau;
#pragma unroll
            for (int t = T0; t < RT; ++t)
#pragma unroll
              for (int v = 0; v < NV; ++v) z[v][t] = fma(a0[v], vr[t], z[v][t]);
          }
        }
      }
    };
    constexpr int TH = RT / 2;         // lane rows before TH: matrix rows before G TH
    const int ch = min(c0 + 1, G * TH / 8);  // stages from ch on touch none of them
    if (c0 >= 0) fetch(c0);
    stages(std::integral_constant<int, TH>{}, c0, ch);
    stages(std::integral_constant<int, 0>{}, ch - 1, 0);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int j = j0 + v * NG + g;
      if (j < kvec) {
#pragma unroll
        for (int t = 0; t < RT; ++t) {
          const int r = gl + G * t;
          if (r < n) Y[(size_t)j * n + r] = z[v][t];
        }
      }
    }
    __syncthreads();
  }
}

// Split by size: the n x kvec block of vectors is spread over the CTA's registers, in as few passes as
// they allow. Beyond 160 the rows a lane holds follow n (12, 14, 16), since two vectors and a reflector of 16 rows no longer fit the
// registers: a molecule of n = 168 takes 13.0 ms against 14.1 with 16 rows, n = 222 29.0 against 30.1. Shared scratch: 16 rows of G RT doubles.
__host__ __device__ constexpr int back_scratch(int n) {
  return 16 * (n <= 32 ? 32 : n <= 64 ? 64 : n <= 96 ? 96 : n <= 128 ? 128 : n <= 160 ? 160 : n <= 192 ? 192 : n <= 224 ? 224 : 256);
}
__device__ __noinline__ void back_transform(int n, int kvec, const double* __restrict__ V, const double* __restrict__ Yt,
                                            double* Y, const EigenScratch& s_) {
  double* sh = in_shared(s_.sh);
  const double* tau = in_shared(s_.tau);
  if (n <= 32) back_transform_t<8, 4, 1>(n, kvec, V, Yt, Y, tau, sh);
  else if (n <= 64 && kvec <= 32) back_transform_t<8, 8, 1>(n, kvec, V, Yt, Y, tau, sh);
  else if (n <= 64) back_transform_t<8, 8, 2>(n, kvec, V, Yt, Y, tau, sh);
  else if (n <= 96) back_transform_t<8, 12, 2>(n, kvec, V, Yt, Y, tau, sh);
  else if (n <= 128 && kvec > 64) back_transform_t<16, 8, 4>(n, kvec, V, Yt, Y, tau, sh);
  else if (n <= 128) back_transform_t<8, 16, 2>(n, kvec, V, Yt, Y, tau, sh);
  else if (n <= 160) back_transform_t<16, 10, 3>(n, kvec, V, Yt, Y, tau, sh);
  else if (n <= 192) back_transform_t<16, 12, 2>(n, kvec, V, Yt, Y, tau, sh);
  else if (n <= 224) back_transform_t<16, 14, 2>(n, kvec, V, Yt, Y, tau, sh);
  else back_transform_t<16, 16, 2>(n, kvec, V, Yt, Y, tau, sh);
}

// All eigenvalues of the saved tridiagonal (d, e) -- used once at the end for the MO energies.
__device__ void all_eigenvalues(int n, const double* d, const double* e, double* out, const EigenScratch& s) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < n; ++i) {
      s.d[i] = d[i];
      s.e[i] = e[i];
    }
  }
  __syncthreads();
  tridiag_eigenvalues(n, n, s);
  for (int j = threadIdx.x; j < n; j += kThreads) out[j] = s.lam[j];
  __syncthreads();
}

}  // namespace pm3gpu
