// rsqrt_f64 (csrc/amk_internal.cuh) of an array, and CUDA's rsqrt beside it.
#include "amk_internal.cuh"

__global__ void rsqrt_kernel(int n, const double* x, double* own, double* cuda) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  own[i] = amk::rsqrt_f64(x[i]);
  cuda[i] = rsqrt(x[i]);
}

// x, own, cuda: n doubles on the host
extern "C" int rsqrt_run(int n, const double* x, double* own, double* cuda) {
  double* d = nullptr;
  const size_t bytes = static_cast<size_t>(n) * sizeof(double);
  if (cudaMalloc(&d, 3 * bytes) != cudaSuccess) return 1;
  int rc = cudaMemcpy(d, x, bytes, cudaMemcpyHostToDevice) != cudaSuccess;
  if (!rc) rsqrt_kernel<<<(n + 255) / 256, 256>>>(n, d, d + n, d + 2 * n);
  rc = rc || cudaMemcpy(own, d + n, bytes, cudaMemcpyDeviceToHost) != cudaSuccess ||
       cudaMemcpy(cuda, d + 2 * n, bytes, cudaMemcpyDeviceToHost) != cudaSuccess;
  cudaFree(d);
  return rc;
}
