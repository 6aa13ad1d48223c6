// exp(x) in double for the Poisson residual's carrier densities, by Tang's
// table-driven method (P. T. P. Tang, "Table-driven implementation of the
// exponential function in IEEE floating-point arithmetic", ACM Trans. Math.
// Softw. 15(2), 1989):
//   x = (256 m + j) ln2/256 + r,  |r| <= ln2/512,
//   exp(x) = 2^m * 2^(j/256) * (1 + p(r)),
// p the Taylor polynomial of e^r - 1 to r^5 (truncation below |r|^6/720 <
// 1e-20 relative).  tab[j] = 2^(j/256), j < 256.  |x| >= 700 and NaN go to the
// library's exp.
// The residual is evaluated in double precision on 16 SMs, whose schedulers issue
// one double instruction of a warp in 64 clocks and one of any other kind in each,
// so only what needs a double's digits is one (five instructions):
//   - k = 256 m + j is rounded in single precision from x cut to a float (any k
//     within a few hundredths of a half serves), by adding 1.5 * 2^23, and made a
//     double by its bits;
//   - r = x - k ln2/256 takes two fused multiply-adds with ln2/256 split into its
//     nearest double and the remainder, so r is accurate to an ulp of r;
//   - c = 1/2 + r/6 + r^2/24 + r^3/120 is formed in fixed point, r as 2^-40 (an
//     error below 2e-13, of a term that r^2 < 2e-6 multiplies), and put together
//     by its bits;  p = r + r^2 c and the table's product are doubles.
// The largest error over |x| < 700 against 64-bit-mantissa exponentials is 1.00
// ulp; nine double instructions with the polynomial to r^4 had 1.33.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define EMCG_HD __host__ __device__ __forceinline__
// (a call, so that the rare path's double instructions are not run beside the other's)
#define EMCG_HD_RARE static __host__ __device__ __noinline__
#else
#define EMCG_HD inline
#define EMCG_HD_RARE inline
#endif

namespace emcg {

constexpr int kExpTab = 256;

EMCG_HD uint64_t dbits(double x) {
  uint64_t b;
  memcpy(&b, &x, sizeof b);
  return b;
}
EMCG_HD double bitsd(uint64_t b) {
  double x;
  memcpy(&x, &b, sizeof x);
  return x;
}

EMCG_HD uint32_t fbits(float x) {
  uint32_t b;
  memcpy(&b, &x, sizeof b);
  return b;
}
EMCG_HD float bitsf(uint32_t b) {
  float x;
  memcpy(&x, &b, sizeof x);
  return x;
}
// the upper 32 bits of the 64-bit product
EMCG_HD int32_t mulHigh(int32_t a, int32_t b) { return (int32_t)(((int64_t)a * b) >> 32); }

EMCG_HD_RARE double expLibrary(double x) { return exp(x); }
EMCG_HD_RARE float floatLibrary(double x) { return (float)x; }

EMCG_HD double expTab(double x, const double *tab) {
  const uint32_t xh = (uint32_t)(dbits(x) >> 32), xl = (uint32_t)dbits(x), xa = xh & 0x7fffffffu;
  // |x| < 700 by the high word of |x| (700 = 0x4085E000 00000000); NaN fails
  if (xa >= 0x4085E000u)
    return expLibrary(x);
  // x cut to a float (below 2^-126: zero); k = 256 m + j, an integer below 2^18
  const float xf =
      bitsf((xh & 0x80000000u) | (xa < 0x38100000u ? 0u : (xa - 0x38000000u) << 3 | xl >> 29));
  const float t = fmaf(xf, 369.32993f, 12582912.f); // x * 256 / ln 2; 1.5 * 2^23
  const int n = (int)(fbits(t) - 0x4b400000u);
  const uint32_t kb = fbits(t - 12582912.f), ka = kb & 0x7fffffffu;
  const double k =
      bitsd((uint64_t)((kb & 0x80000000u) | (ka ? (ka >> 3) + 0x38000000u : 0u)) << 32);
  const double r = fma(-k, 9.058776616587108e-20, fma(-k, 0.0027076061740622863, x));
  // r in 2^-40: |r| < 2^-9
  const uint32_t rh = (uint32_t)(dbits(r) >> 32), rl = (uint32_t)dbits(r);
  const uint32_t mant = (rh & 0xfffffu) << 11 | 0x80000000u | rl >> 21;
  const int sh = 1014 - (int)(rh >> 20 & 0x7ffu); // at least 1
  const int32_t ra = (int32_t)(mant >> (sh < 31 ? sh : 31));
  const int32_t R = (int32_t)rh < 0 ? -ra : ra;
  const int32_t v2 = 1431655765 + mulHigh(R, 1118481);        // 1/24 + r/120 in 2^-35
  const int32_t v1 = 1431655765 + (mulHigh(R, v2) >> 10);     // 1/6 + r/24 + r^2/120 in 2^-33
  const int64_t d = ((int64_t)R * v1) >> 20;                  // times r, in 2^-53
  // 1/2 + d: below 1/2 a unit of the last place is half as large
  const double c = bitsd(0x3FE0000000000000ull + (uint64_t)(d < 0 ? 2 * d : d));
  const double p = fma(r * r, c, r);
  const double T = tab[n & (kExpTab - 1)];
  const double y = fma(T, p, T);
  // y * 2^m, m = (n - j) / 256: y is near 1, the result stays normal
  return bitsd(dbits(y) + ((uint64_t)(uint32_t)((n >> 8) << 20) << 32));
}

// x rounded to a float (to nearest, ties to even) and v as a double, by their bits:
// the conversions' instructions run at the double-precision rate.  Values beyond
// the floats' normal range, zeros and NaN go to the conversions.
EMCG_HD float toFloat(double x) {
  const uint32_t h = (uint32_t)(dbits(x) >> 32), l = (uint32_t)dbits(x), a = h & 0x7fffffffu;
  if (a - 0x38100000u >= 0x47e00000u - 0x38100000u) // 2^-126 <= |x| < 2^127
    return floatLibrary(x);
  const uint32_t v = (a - 0x38000000u) << 3 | l >> 29;
  return bitsf((h & 0x80000000u) | (v + (((l & 0x1fffffffu) + 0x0fffffffu + (v & 1u)) >> 29)));
}
EMCG_HD double toDouble(float v) {
  const uint32_t b = fbits(v), a = b & 0x7fffffffu;
  if (a - 0x00800000u >= 0x7f800000u - 0x00800000u)
    return (double)v;
  return bitsd((uint64_t)((b & 0x80000000u) | ((a >> 3) + 0x38000000u)) << 32 |
               (uint64_t)(a << 29));
}

} // namespace emcg
