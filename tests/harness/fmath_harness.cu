// The functions of fmath.cuh on arrays, for tests/test_fmath.py: exp, log and
// x^y in the host compilation of the same source and on the device, the
// reciprocal and the quotient (seeded by the device's special-function unit)
// on the device.
#include "../../phd_gb300/csrc/fmath.cuh"

namespace {
__global__ void k_apply(int op, long long n, const double* a, const double* b, double* y) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  switch (op) {
    case 0: y[i] = fm_exp(a[i]); break;
    case 1: y[i] = fm_log(a[i]); break;
    case 2: y[i] = fm_root(a[i], b[i]); break;
    case 3: y[i] = fm_rcp(a[i]); break;
    default: y[i] = fm_div(a[i], b[i]);
  }
}
}  // namespace

extern "C" int fmath_host(int op, long long n, const double* a, const double* b, double* y) {
  for (long long i = 0; i < n; ++i) {
    switch (op) {
      case 0: y[i] = fm_exp(a[i]); break;
      case 1: y[i] = fm_log(a[i]); break;
      case 2: y[i] = fm_root(a[i], b[i]); break;
      default: return 1;
    }
  }
  return 0;
}

extern "C" int fmath_device(int op, long long n, const double* a, const double* b, double* y) {
  double *da = nullptr, *db = nullptr, *dy = nullptr;
  int rc = 1;
  if (!cudaMalloc(&da, n * 8) && !cudaMalloc(&db, n * 8) && !cudaMalloc(&dy, n * 8) &&
      !cudaMemcpy(da, a, n * 8, cudaMemcpyHostToDevice) && !cudaMemcpy(db, b, n * 8, cudaMemcpyHostToDevice)) {
    k_apply<<<(unsigned)((n + 255) / 256), 256>>>(op, n, da, db, dy);
    if (!cudaGetLastError() && !cudaMemcpy(y, dy, n * 8, cudaMemcpyDeviceToHost)) rc = 0;
  }
  cudaFree(da);
  cudaFree(db);
  cudaFree(dy);
  return rc;
}
