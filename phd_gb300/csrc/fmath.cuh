// FP64 elementary functions off the FP64 pipe.
//
// The GB300 SM starts two FP64 operations a clock (measured 1.96) and 128
// 32-bit ones, and the division, reciprocal, exponential and logarithm of
// the CUDA library are chains of FP64 operations: measured in slots of that
// pipe, 1/x takes 5.4, a/x 9, exp 19 and log 36.  The functions here take a
// seed from the special-function unit and as few FP64 operations as reach
// the rounding of the format.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

// true when |x| is in [2^-900, 2^900): the seed, its square and the products
// below then neither overflow nor lose bits to underflow
__device__ __forceinline__ bool fm_mid(double x) {
  const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
  return e - 123u < 1800u;
}

// 2^-20-accurate reciprocal (special-function unit, PTX rcp.approx.ftz.f64)
__device__ __forceinline__ double fm_rcp_seed(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}

// 1 / x: one third-order step y (1 + e + e^2), e = 1 - x y, from the seed
// (truncation |e|^3 < 2^-57).  3 slots against 5.4 of 1.0 / x.
__device__ __forceinline__ double fm_rcp(double x) {
  if (!fm_mid(x)) return 1.0 / x;
  const double y = fm_rcp_seed(x);
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// a / x: a second-order step on the seed, the quotient, and its exact
// remainder folded back (truncation |e|^4).  5 slots against 9 of a / x.
__device__ __forceinline__ double fm_div(double a, double x) {
  const unsigned ea = ((unsigned)__double2hiint(a) >> 20) & 0x7ffu;
  const unsigned ex = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
  // the quotient and the remainder stay normal (a = 0 takes the general form)
  if (!(ex - 523u < 1000u) || !(ea - 523u < 1000u)) return a / x;
  double y = fm_rcp_seed(x);
  y = fma(y, fma(-x, y, 1.0), y);
  const double q = a * y;
  return fma(fma(-x, q, a), y, q);
}
