// The parts of the double-precision building blocks (emcg_fp64.cuh) that need no
// GPU instruction: comparisons and conversions by bit patterns, and the steps
// from the hardware's approximations to full precision.
#pragma once

#include <math.h>

#include "emcg_exp.h" // EMCG_HD, dbits, bitsd

namespace emcg {

// 1 / sqrt(t) from the hardware's approximation y (relative error measured 1.01 x
// 2^-20): one step of Householder's method of third order (Householder 1970), with
// e = 1 - t y^2, y (1 + e / 2 + 3 e^2 / 8).  y has 20 fraction bits, so y y is exact
// and e is rounded once, at its own size: the result is within 0.53 units in the
// last place (0.5 for the last addition, 0.02 for 5 e^3 / 16; 1.03 with e as
// 1 - (t y) y), against 0.85 of a division and a square root.
EMCG_HD double rsqrtStep(double t, double y) {
  const double e = fma(-t, y * y, 1.0);
  return fma(fma(0.375, e, 0.5), y * e, y);
}

// 1 / d from such a y: y (1 + r + r^2), r = 1 - d y (the geometric series to third
// order); within 0.52 units in the last place
EMCG_HD double rcpStep(double d, double y) {
  const double r = fma(-d, y, 1.0);
  return fma(y, fma(r, r, r), y);
}

// a < b for a double a and b >= 0 without a double-precision instruction: the
// bit patterns of non-negative doubles order like the values, those of
// negative ones are negative integers; -0 counts as 0, and a NaN is not below
EMCG_HD bool belowD(double a, double b) {
  const int64_t x = (int64_t)dbits(a), y = (int64_t)dbits(b);
  return (x == INT64_MIN ? 0 : x) < y && (uint64_t)x <= 0xfff0000000000000ull;
}

// a < 0 and a <= 0 the same way
EMCG_HD bool negativeD(double a) {
  return dbits(a) - 0x8000000000000001ull <= 0x7fefffffffffffffull;
}
EMCG_HD bool notPositiveD(double a) {
  return (int64_t)dbits(a) <= 0 && dbits(a) <= 0xfff0000000000000ull;
}

// q as an integer part and 20 fractional bits, for 0 <= q < 2^30; false outside
EMCG_HD bool fixedOf(double q, uint64_t &f) {
  const uint64_t b = dbits(q);
  const int e = (int)(b >> 52) - 1023;
  if (e >= 30) // also a negative q, infinities and NaN
    return false;
  const uint64_t mant = (b & 0xfffffffffffffull) | 0x10000000000000ull;
  f = e < -31 ? 0 : mant >> (32 - e);
  return true;
}

} // namespace emcg
