// Pieces of the per-CTA eigensolver by themselves, for tests/test_gpu_eigen_pieces.py.
#include "cta_eigen.cuh"

using namespace pm3gpu;

// The lowest kval eigenvalues of a tridiagonal (n <= 256), one CTA.
__global__ void __launch_bounds__(kThreads) eigenvalues_kernel(int n, int kval, const double* d, const double* e, double* lam) {
  extern __shared__ __align__(16) unsigned char smem[];
  double* p = reinterpret_cast<double*>(smem);
  EigenScratch s{};
  s.red = p;
  s.misc = p + 8 * kWarps;
  p += 8 * kWarps + 8;
  s.d = p;
  s.e = p + n;
  s.e2 = p + 2 * n;
  s.lam = p + 3 * n;
  s.blk = reinterpret_cast<int*>(p + 4 * n);
  s.nblk = s.blk + n + 1;
  for (int i = threadIdx.x; i < n; i += kThreads) {
    s.d[i] = d[i];
    s.e[i] = e[i];
  }
  __syncthreads();
  tridiag_eigenvalues(n, kval, s);
  for (int j = threadIdx.x; j < kval; j += kThreads) lam[j] = s.lam[j];
}

extern "C" int probe_eigenvalues(int n, int kval, const double* d, const double* e, double* lam) {
  if (n < 1 || n > kMaxN || kval < 1 || kval > n) return -1;
  double* b = nullptr;
  if (cudaMalloc(&b, 3 * n * sizeof(double)) != cudaSuccess) return 1;
  cudaMemcpy(b, d, n * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(b + n, e, n * sizeof(double), cudaMemcpyHostToDevice);
  const size_t bytes = (8 * kWarps + 8 + 4 * n) * sizeof(double) + (n + 2) * sizeof(int);
  eigenvalues_kernel<<<1, kThreads, bytes>>>(n, kval, b, b + n, b + 2 * n);
  cudaMemcpy(lam, b + 2 * n, kval * sizeof(double), cudaMemcpyDeviceToHost);
  const int rc = (int)cudaDeviceSynchronize();
  cudaFree(b);
  return rc;
}

// Largest differences, in units of the last place, of sqrt_newton and rcp_newton from CUDA's square root and division: every
// exponent from -797 to 796 (1e-240 to 1e239), `each` random mantissas of one and the two ends of the binade.
__global__ void roots_kernel(int each, unsigned long long* out) {
  const int ex = (int)blockIdx.x - 797;
  unsigned long long s = 0x9e3779b97f4a7c15ull * (blockIdx.x * blockDim.x + threadIdx.x + 1), m0 = 0, m1 = 0;
  for (int i = threadIdx.x; i < each + 4; i += blockDim.x) {
    s = s * 6364136223846793005ull + 1442695040888963407ull;
    unsigned long long t = s ^ (s >> 29);
    t = (t * 0xbf58476d1ce4e5b9ull) >> 12;  // 52 bits
    if (i < 4) t = i < 2 ? (unsigned long long)i : (1ull << 52) - (unsigned long long)(i - 1);
    const double x = __longlong_as_double(((long long)(ex + 1023) << 52) | (long long)t);
    const long long a = __double_as_longlong(sqrt_newton(x)) - __double_as_longlong(sqrt(x));
    const long long b = __double_as_longlong(rcp_newton(x)) - __double_as_longlong(1.0 / x);
    m0 = max(m0, (unsigned long long)llabs(a));
    m1 = max(m1, (unsigned long long)llabs(b));
  }
  atomicMax(out, m0);
  atomicMax(out + 1, m1);
}

extern "C" int probe_roots(int each, unsigned long long* out) {
  unsigned long long* b = nullptr;
  if (cudaMalloc(&b, 16) != cudaSuccess) return 1;
  cudaMemset(b, 0, 16);
  roots_kernel<<<797 + 797, 256>>>(each, b);
  cudaMemcpy(out, b, 16, cudaMemcpyDeviceToHost);
  const int rc = (int)cudaDeviceSynchronize();
  cudaFree(b);
  return rc;
}
