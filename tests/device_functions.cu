// Device functions of the library, one thread per argument, for test_device_functions.py.
#include "../pytential_b200/csrc/helmholtz.cuh"

namespace {

__global__ void k_y01(int n, const double* x, double* y0, double* y1)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) qbx::bessel_y01(x[i], y0[i], y1[i]);
}

__global__ void k_rsqrt(int n, const double* x, double* seed, double* h, double* lib)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x[i]));
  seed[i] = y;
  h[i] = qbx::rsqrt_h(x[i]);
  lib[i] = rsqrt(x[i]);
}

}  // namespace

extern "C" {

int device_y01(int n, const double* x, double* y0, double* y1, void* stream)
{
  k_y01<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(n, x, y0, y1);
  return cudaGetLastError();
}

int device_rsqrt(int n, const double* x, double* seed, double* h, double* lib, void* stream)
{
  k_rsqrt<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(n, x, seed, h, lib);
  return cudaGetLastError();
}

}  // extern "C"
