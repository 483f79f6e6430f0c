// The dense solves of dwsolve.cuh on systems from the host, one CTA of 128
// threads per system (n <= 16 rows, at most 16 right-hand sides): the FP32
// inverse with the right-hand sides refined (refine_any), the corrected
// double-word inverse (correct_inverse) and the double-word LDL^T.
#include <cuda_runtime.h>

#include "dwsolve.cuh"

using namespace mlcp;

namespace {

constexpr int kMax = 16;

__device__ void put(const dw* x, double* out, int count) {
  for (int e = threadIdx.x; e < count; e += blockDim.x) out[e] = dw_to_double(x[e]);
}

// A [n][n], B and the solutions [nrhs][n] per system; solved and cycles: [3] each.
__global__ void __launch_bounds__(dwsolve::kSolverThreads) check_kernel(int n, int nrhs, const double* A, const double* B,
                                                                       double* X, int* solved, long long* cycles) {
  __shared__ dw a[kMax * kMax], b[kMax * kMax], x[kMax * kMax], iv[kMax * kMax], res[kMax * kMax], dinv[kMax], u[kMax];
  __shared__ float gi[kMax * kMax], ef[kMax * kMax], emax[dwsolve::kSolverWarps], red[4];
  __shared__ int good;
  const int t = threadIdx.x, nn = n * n, nr = n * nrhs;
  const size_t sys = blockIdx.x;
  for (int e = t; e < nn; e += blockDim.x) a[e] = dw_from_double(A[sys * nn + e]);
  for (int e = t; e < nr; e += blockDim.x) b[e] = dw_from_double(B[sys * nr + e]);
  __syncthreads();
  if (t < 32) {
    const bool g = dwsolve::gj_inverse_warp(a, n, gi);
    if (t == 0) good = g;
  }
  __syncthreads();
  double* out = X + sys * 3 * nr;
  long long c0 = clock64();
  bool ok = good && dwsolve::refine_any<dwsolve::kSolverThreads>(a, n, b, x, nrhs, gi, res, red);
  __syncthreads();
  long long c1 = clock64();
  if (t == 0) {
    solved[sys * 3] = ok;
    cycles[sys * 3] = c1 - c0;
  }
  put(x, out, nr);
  __syncthreads();
  c0 = clock64();
  ok = good && dwsolve::correct_inverse<0>(a, n, gi, iv, ef, emax);
  __syncthreads();
  c1 = clock64();
  if (t == 0) {
    solved[sys * 3 + 1] = ok;
    cycles[sys * 3 + 1] = c1 - c0;
  }
  for (int e = t; ok && e < nr; e += blockDim.x) {
    const int i = e % n, m = e / n;
    dw_acc acc = acc_zero();
    for (int k = 0; k < n; ++k) acc_fma(acc, iv[i + k * n], b[k + m * n]);
    x[e] = acc_value(acc);
  }
  __syncthreads();
  put(x, out + nr, nr);
  __syncthreads();
  for (int e = t; e < nr; e += blockDim.x) x[e] = b[e];
  __syncthreads();
  c0 = clock64();
  const int bad = dwsolve::dw_ldlt(a, n, dinv, u);
  dwsolve::dw_ldlt_solve(a, n, dinv, x, nrhs);
  __syncthreads();
  c1 = clock64();
  if (t == 0) {
    solved[sys * 3 + 2] = bad == 0;
    cycles[sys * 3 + 2] = c1 - c0;
  }
  put(x, out + 2 * nr, nr);
}

}  // namespace

// Host arrays in and out; 0 on success, 1 for sizes that the kernel does not take, else a CUDA error.
extern "C" int dwsolve_check(int n, int nrhs, int nsys, const double* A, const double* B, double* X, int* solved,
                             long long* cycles) {
  if (n < 1 || n > kMax || nrhs < 1 || nrhs > kMax || nsys < 1) return 1;
  const size_t nn = (size_t)n * n * nsys, nr = (size_t)n * nrhs * nsys;
  double *dA = nullptr, *dB = nullptr, *dX = nullptr;
  int* ds = nullptr;
  long long* dc = nullptr;
  cudaError_t rc = cudaMalloc(&dA, sizeof(double) * nn);
  if (!rc) rc = cudaMalloc(&dB, sizeof(double) * nr);
  if (!rc) rc = cudaMalloc(&dX, sizeof(double) * 3 * nr);
  if (!rc) rc = cudaMalloc(&ds, sizeof(int) * 3 * nsys);
  if (!rc) rc = cudaMalloc(&dc, sizeof(long long) * 3 * nsys);
  if (!rc) rc = cudaMemcpy(dA, A, sizeof(double) * nn, cudaMemcpyHostToDevice);
  if (!rc) rc = cudaMemcpy(dB, B, sizeof(double) * nr, cudaMemcpyHostToDevice);
  if (!rc) {
    check_kernel<<<nsys, dwsolve::kSolverThreads>>>(n, nrhs, dA, dB, dX, ds, dc);
    rc = cudaGetLastError();
  }
  if (!rc) rc = cudaMemcpy(X, dX, sizeof(double) * 3 * nr, cudaMemcpyDeviceToHost);
  if (!rc) rc = cudaMemcpy(solved, ds, sizeof(int) * 3 * nsys, cudaMemcpyDeviceToHost);
  if (!rc) rc = cudaMemcpy(cycles, dc, sizeof(long long) * 3 * nsys, cudaMemcpyDeviceToHost);
  cudaFree(dA);
  cudaFree(dB);
  cudaFree(dX);
  cudaFree(ds);
  cudaFree(dc);
  return (int)rc;
}
