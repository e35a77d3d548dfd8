// The force terms' roots and the CUDA library's, element by element.
#include "forces.cuh"

__global__ void k_roots(const double *x, int n, double *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = ladds::rsqrtOf(x[i]);
  out[n + i] = ladds::sqrtOf(x[i]);
  out[2 * n + i] = rsqrt(x[i]);
  out[3 * n + i] = sqrt(x[i]);
}

// out: four rows of n; returns a CUDA error code
extern "C" int roots(const double *x, int n, double *out) {
  double *d = nullptr;
  cudaError_t e = cudaMalloc(&d, 5 * (size_t)n * sizeof(double));
  if (e != cudaSuccess) return (int)e;
  e = cudaMemcpy(d, x, (size_t)n * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_roots<<<(n + 255) / 256, 256>>>(d, n, d + n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d + n, 4 * (size_t)n * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
