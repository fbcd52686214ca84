// The FP64 1/sqrt of the pair kernels and CUDA's own over an array, for
// tests/test_gpu_rsqrt64.py: out is [3][n], rsqrt_f64, rsqrt_f64_full and rsqrt.
#include "rsqrt64.cuh"

__global__ void all_of(const double *x, double *out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = pawan::rsqrt_f64(x[i]);
  out[n + i] = pawan::rsqrt_f64_full(x[i]);
  out[2 * (size_t)n + i] = rsqrt(x[i]);
}

extern "C" int rsqrt64_probe(const double *x, double *out, int n) {
  if (n <= 0) return 0;
  all_of<<<(n + 255) / 256, 256>>>(x, out, n);
  return (int)cudaDeviceSynchronize();
}
