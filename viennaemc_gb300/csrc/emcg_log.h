// log(x) in double for the free-flight draws, by Tang's table-driven method
// (P. T. P. Tang, "Table-driven implementation of the logarithm function in IEEE
// floating-point arithmetic", ACM Trans. Math. Softw. 16(4), 1990):
//   x = 2^e m,  11/16 <= m < 11/8,  r = m c_j - 1 with c_j near 1 / m,
//   log(x) = e ln2 - log(c_j) + log1p(r),
// 128 intervals of m, log1p(r) by its Taylor polynomial to r^8 (|r| <= 1/128:
// truncation below 2^-59 relative).  The two intervals beside 1 have c = 1, so
// that r = x - 1 is exact there and the result keeps its relative accuracy as
// x goes to 1.  e ln2 comes from a table of its leading part and the rest.
// Both table sums are split into a leading part of at most 46 bits and the
// rest, so the leading parts add without rounding.  Arguments outside
// [2^-30, 11/8) go to the library's log.  14 double-precision instructions: the
// double pipe bounds the step kernel that draws with it.
#pragma once

#include "emcg_exp.h" // EMCG_HD, dbits, bitsd

namespace emcg {

constexpr int kLogIntervals = 128;
constexpr int kLogExps = 32;
// the table: c_j and the leading part of -log(c_j) per interval, the leading
// part and the rest of -k ln2 for k = 0 .. kLogExps - 1, and the rest of
// -log(c_j) per interval
constexpr int kLogTab = 3 * kLogIntervals + 2 * kLogExps;

// x to a multiple of 2^-40 (|x| < 2^11)
inline double logLead(double x) { return (x + 6144.0) - 6144.0; }

// entry i of the table, formed on the host in extended precision
inline double logTabEntry(int i) {
  const double ln2Hi = 0.6931471805599453, ln2Lo = 2.3190468138462996e-17;
  const bool exps = i >= 2 * kLogIntervals && i < 2 * kLogIntervals + 2 * kLogExps;
  if (exps) {
    const int k = (i - 2 * kLogIntervals) / 2;
    const double lead = -k * logLead(ln2Hi); // 40 + 5 bits: exact
    return i & 1 ? -k * (ln2Hi - logLead(ln2Hi)) - k * ln2Lo : lead;
  }
  const int j = i < 2 * kLogIntervals ? i / 2 : i - 2 * kLogIntervals - 2 * kLogExps;
  // the interval's bounds by their high words
  const double a = bitsd((uint64_t)(0x3fe60000u + (uint32_t)j * 0x2000u) << 32);
  const double b = bitsd((uint64_t)(0x3fe60000u + (uint32_t)(j + 1) * 0x2000u) << 32);
  const double c = a == 1.0 || b == 1.0 ? 1.0 : 2.0 / (a + b);
  if (i < 2 * kLogIntervals && !(i & 1))
    return c;
  const long double l = -logl((long double)c);
  const double lead = logLead((double)l);
  return i < 2 * kLogIntervals ? lead : (double)(l - (long double)lead);
}

EMCG_HD double logTab(double x, const double *tab) {
  const uint64_t b = dbits(x);
  const uint32_t h = (uint32_t)(b >> 32);
  if (h - 0x3e100000u >= 0x3ff60000u - 0x3e100000u) // not in [2^-30, 11/8)
    return log(x);
  const int e = (int)(h - 0x3fe60000u) >> 20;
  const uint32_t hm = h - ((uint32_t)e << 20);
  const double m = bitsd((uint64_t)hm << 32 | (uint32_t)b);
  const int j = (int)((hm - 0x3fe60000u) >> 13);
  const int k = -e; // 0 .. 30
  const double r = fma(m, tab[2 * j], -1.0);
  double q = fma(r, -1.0 / 8, 1.0 / 7);
  q = fma(r, q, -1.0 / 6);
  q = fma(r, q, 1.0 / 5);
  q = fma(r, q, -1.0 / 4);
  q = fma(r, q, 1.0 / 3);
  q = fma(r, q, -1.0 / 2);
  const double *te = tab + 2 * kLogIntervals + 2 * k;
  const double t = te[1] + tab[2 * kLogIntervals + 2 * kLogExps + j];
  return (te[0] + tab[2 * j + 1]) + fma(r * r, q, r + t);
}

} // namespace emcg
