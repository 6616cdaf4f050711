// The mixed path's quotient and reciprocal on given operands (host arrays).
#include "rfgpu_kernels.cuh"

namespace rfgpu {
__global__ void k_check(const float *a, const float *b, int n, float *quot, float *rec) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  quot[i] = venkat_div(a[i], b[i]);
  rec[i] = rcp_ftz(b[i]);
}
}  // namespace rfgpu

extern "C" int reciprocal_check(const float *a, const float *b, int n, float *quot, float *rec) {
  float *d = nullptr;
  const size_t s = (size_t)n * sizeof(float);
  if (cudaMalloc(&d, 4 * s) != cudaSuccess) return 1;
  cudaMemcpy(d, a, s, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b, s, cudaMemcpyHostToDevice);
  rfgpu::k_check<<<(n + 255) / 256, 256>>>(d, d + n, n, d + 2 * (size_t)n, d + 3 * (size_t)n);
  cudaMemcpy(quot, d + 2 * (size_t)n, s, cudaMemcpyDeviceToHost);
  cudaMemcpy(rec, d + 3 * (size_t)n, s, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
