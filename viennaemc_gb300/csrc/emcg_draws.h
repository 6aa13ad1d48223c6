// The double engine's uniform draw and table level with few double-precision
// instructions, of which a GB300 SM issues one in the time of about 70 integer
// ones: the same results as the plain expressions, bit for bit.
#pragma once

#include "emcg_exp.h" // EMCG_HD, dbits, bitsd

namespace emcg {

// (double)w / 2^64 rounded to nearest even, clamped below 1 (libstdc++'s
// generate_canonical<double, 53> of one 64-bit word), in integers
EMCG_HD double canonicalBits(uint64_t w) {
  if (w == 0)
    return 0.0;
#ifdef __CUDA_ARCH__
  const int lz = __clzll((long long)w);
#else
  const int lz = __builtin_clzll(w);
#endif
  const uint64_t m = w << lz;
  uint64_t q = m >> 11;
  const uint32_t rest = (uint32_t)m & 0x7ffu;
  q += rest > 0x400u || (rest == 0x400u && (q & 1)) ? 1 : 0;
  // q in [2^52, 2^53]: its leading bit (or the carry to 2^53) adds to the exponent
  const uint64_t bits = ((uint64_t)(1021 - lz) << 52) + q;
  return bitsd(bits >= 0x3ff0000000000000ull ? 0x3fefffffffffffffull : bits);
}

// The table level of energy E (include/emcScatterHandler.hpp:237-244): floor(E / dE)
// - 1 with the reference's size_t conversion, -1 giving 0, other negative
// values, NaN and what lies above the table the top level.
EMCG_HD int levelExact(double E, double dE, int nLevels) {
  const double f = floor(E / dE) - 1;
  if (!(f >= 0.))
    return f == -1. ? 0 : nLevels - 1;
  return f > (double)(nLevels - 1) ? nLevels - 1 : (int)f;
}

// The same by one multiplication: the quotient's integer part from its bits.
// A quotient within 8 units in the last place of a whole number, where
// E * (1 / dE) and E / dE may fall on either side of it, is divided exactly.
EMCG_HD int levelFast(double E, double dE, double invdE, int nLevels) {
  const double q = E * invdE;
  const uint64_t b = dbits(q);
  const int e = (int)(b >> 52) - 1023; // a negative or not finite q gives e >= 31
  if (e >= 0 && e < 31) {
    const uint64_t mant = (b & 0xfffffffffffffull) | 0x10000000000000ull;
    const uint64_t fr = mant & ((1ull << (52 - e)) - 1);
    if (fr >= 8 && fr + 8 <= (1ull << (52 - e))) {
      const int f = (int)(mant >> (52 - e)) - 1;
      return f > nLevels - 1 ? nLevels - 1 : f;
    }
  } else if (e < 0 && b + 8 <= 0x3ff0000000000000ull) {
    return 0; // 0 <= E / dE < 1: level -1
  }
  return levelExact(E, dE, nLevels);
}

} // namespace emcg
