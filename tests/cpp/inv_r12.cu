// invR12 (csrc/common.cuh) on an array, for tests/test_gpu_inv_r12.py.
#include "common.cuh"

__global__ void kInvR12(int64_t n, const double * x, double * y)
{
  int64_t const i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i < n) y[i] = tcscf::invR12(x[i]);
}

extern "C" int inv_r12(int64_t n, const double * x, double * y)
{
  double * d = nullptr;
  if (cudaMalloc(&d, sizeof(double) * 2 * n) != cudaSuccess) return 1;
  cudaMemcpy(d, x, sizeof(double) * n, cudaMemcpyHostToDevice);
  kInvR12<<<unsigned((n + 255) / 256), 256>>>(n, d, d + n);
  cudaError_t const e = cudaMemcpy(y, d + n, sizeof(double) * n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? 0 : 2;
}
