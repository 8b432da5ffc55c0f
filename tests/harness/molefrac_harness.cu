// The shared reciprocal of a point's mole fractions (fmath.cuh) on arrays, for
// tests/test_gpu_molefrac.py.
#include "../../phd_gb300/csrc/fmath.cuh"

namespace {
__global__ void k_apply(int n, const double* x, const double* a, const double* b, double* y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = fm_over(x[i], fm_rcp_prod(a[i], b[i]));
}
}  // namespace

extern "C" int molefrac_device(int n, const double* x, const double* a, const double* b, double* y) {
  double* d = nullptr;
  const size_t s = (size_t)n * sizeof(double);
  int rc = 1;
  if (!cudaMalloc(&d, 4 * s) && !cudaMemcpy(d, x, s, cudaMemcpyHostToDevice) &&
      !cudaMemcpy(d + n, a, s, cudaMemcpyHostToDevice) && !cudaMemcpy(d + 2 * (size_t)n, b, s, cudaMemcpyHostToDevice)) {
    k_apply<<<(n + 255) / 256, 256>>>(n, d, d + n, d + 2 * (size_t)n, d + 3 * (size_t)n);
    if (!cudaGetLastError() && !cudaMemcpy(y, d + 3 * (size_t)n, s, cudaMemcpyDeviceToHost)) rc = 0;
  }
  cudaFree(d);
  return rc;
}
