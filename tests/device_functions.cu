// Device functions of the library, one thread per argument, for test_device_functions.py.
#include "../pytential_b200/csrc/helmholtz.cuh"

namespace {

__global__ void k_y01(int n, const double* x, double* y0, double* y1)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) qbx::bessel_y01(x[i], y0[i], y1[i]);
}

}  // namespace

extern "C" {

int device_y01(int n, const double* x, double* y0, double* y1, void* stream)
{
  k_y01<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(n, x, y0, y1);
  return cudaGetLastError();
}

}  // extern "C"
