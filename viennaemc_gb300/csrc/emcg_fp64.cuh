// Double-precision building blocks for a GPU whose schedulers issue one double
// instruction of a warp in 64 clocks: square root, reciprocal and quotient from
// the hardware's approximations with one correction each.  The results are the
// correctly rounded ones or their neighbours; sqrtD and divD hand arguments outside
// their range to the library.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "emcg_fp64.h"

namespace emcg {

// 1 / sqrt(t) for normal t > 0, and 1 / d for normal d whose reciprocal is normal
// (the caller's to see to: neither has another path)
__device__ __forceinline__ double rsqrtD(double t) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(t));
  return rsqrtStep(t, y);
}
__device__ __forceinline__ double rcpD(double d) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  return rcpStep(d, y);
}

// sqrt(x): x / sqrt(x) corrected once; 0, subnormals, infinities, negative
// values and NaN go to the library's
__device__ __forceinline__ double sqrtD(double x) {
  const uint32_t h = (uint32_t)__double2hiint(x);
  if (h - 0x00100000u >= 0x7fe00000u)
    return sqrt(x);
  const double y = rsqrtD(x), s = x * y;
  return fma(fma(-s, s, x), 0.5 * y, s);
}

// a / b: a times 1 / b corrected once; where an exponent is near the range's
// ends the library's division
__device__ __forceinline__ double divD(double a, double b) {
  const uint32_t ha = (uint32_t)__double2hiint(a) & 0x7fffffffu,
                 hb = (uint32_t)__double2hiint(b) & 0x7fffffffu;
  // both in [2^-500, 2^500]
  if (ha - 0x20b00000u >= 0x3e800000u || hb - 0x20b00000u >= 0x3e800000u)
    return a / b;
  const double inv = rcpD(b), q = a * inv;
  return fma(fma(-b, q, a), inv, q);
}

} // namespace emcg
