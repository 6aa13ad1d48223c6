// The parts of the double-precision building blocks (emcg_fp64.cuh) that need no
// GPU instruction: comparisons and conversions by bit patterns.
#pragma once

#include "emcg_exp.h" // EMCG_HD, dbits, bitsd

namespace emcg {

// a < b for a double a and b >= 0 without a double-precision instruction: the
// bit patterns of non-negative doubles order like the values, those of
// negative ones are negative integers; -0 counts as 0, and a NaN is not below
EMCG_HD bool belowD(double a, double b) {
  const int64_t x = (int64_t)dbits(a), y = (int64_t)dbits(b);
  return (x == INT64_MIN ? 0 : x) < y && (uint64_t)x <= 0xfff0000000000000ull;
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
