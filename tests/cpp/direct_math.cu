// The pair kernel's reciprocal beside CUDA's division, for tests/test_gpu_direct_math.py.
#include <cuda_runtime.h>

#include "pme_direct_math.h"

__global__ void k_reciprocal(const double* x, int n, double* guess_error, double* mine, double* division) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  guess_error[i] = __fma_rn(-x[i], pme::direct::reciprocal_guess(x[i]), 1.0);
  mine[i] = pme::direct::reciprocal(x[i]);
  division[i] = 1.0 / x[i];
}

// device arrays of n doubles each; the CUDA status
extern "C" int reciprocal_run(const double* x, int n, double* guess_error, double* mine, double* division) {
  if (n <= 0) return 0;
  k_reciprocal<<<(n + 255) / 256, 256>>>(x, n, guess_error, mine, division);
  const cudaError_t e = cudaGetLastError();
  return (int)(e == cudaSuccess ? cudaDeviceSynchronize() : e);
}
