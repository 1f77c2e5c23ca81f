// the library's reciprocals and roots, elementwise (test_gpu_reciprocals.py compiles this)
#include "fos_device.cuh"

__global__ void k_recips(long n, const double* __restrict__ x, double* __restrict__ out) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double root;
  out[i] = rcp64(x[i]);
  out[n + i] = rsqrt64(x[i], root);
  out[2 * n + i] = root;
  out[3 * n + i] = rcp64_normal(x[i]);
}

extern "C" int recips(long n, const double* x, double* out) {
  k_recips<<<(unsigned)((n + 255) / 256), 256>>>(n, x, out);
  const cudaError_t e = cudaDeviceSynchronize();
  return e == cudaSuccess ? (int)cudaGetLastError() : (int)e;
}
