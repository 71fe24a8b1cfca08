// Reciprocals and roots of the FP64 factorisation's pivots, which sit on its
// chain of eliminations: from the hardware's approximations by published
// iterations, a few dependent FP64 operations each, where the division and the
// root take a subroutine.  Within one unit in the last place of the exact
// value (tests/test_pivot_math.py).
#pragma once
#include <cuda_runtime.h>

namespace gbba {

// 2^-900 <= d < 2^900: every intermediate value below is a normal number.  The
// approximations flush subnormal arguments and results to zero, so pivots
// outside go through the division and the root.
__device__ __forceinline__ bool plain_range(double d) {
  return (unsigned)__double2hiint(d) - 0x07b00000u < 0x78300000u - 0x07b00000u;
}

// 1 / d from the hardware's approximate reciprocal r: with e = 1 - d r, the
// next terms of the geometric series 1 / d = r (1 + e + e^2 + ...) (Newton's
// iteration of third order).
__device__ __forceinline__ double rcp_series(double d) {
  if (!plain_range(d)) return 1.0 / d;
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  const double e = fma(-d, r, 1.0);
  return fma(r, fma(e, e, e), r);
}
// s = sqrt(d) and r = 1 / s: two of Newton's steps y += y (1 - d y^2) / 2 from
// the hardware's approximation of 1 / sqrt(d), then s = d y and r = y with a
// last step each, so that s r = 1 to rounding.
__device__ __forceinline__ void sqrt_newton(double d, double& s, double& r) {
  if (!plain_range(d)) {
    s = sqrt(d);
    r = 1.0 / s;
    return;
  }
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const double e = fma(-d * y, y, 1.0);
    y = fma(0.5 * y, e, y);
  }
  s = d * y;
  s = fma(0.5 * y, fma(-s, s, d), s);
  r = fma(y, fma(-s, y, 1.0), y);
}
__device__ __forceinline__ bool positive_finite(double d) {  // on the bits: FP64 comparisons run on the FP64 pipe
  const unsigned hi = (unsigned)__double2hiint(d);
  return hi < 0x7ff00000u && (hi | (unsigned)__double2loint(d)) != 0u;
}

}  // namespace gbba
