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
