// emcg::toFloat and emcg::toDouble against the conversions, bit for bit: random
// bit patterns, exponents around the floats' range, ties and their neighbours,
// zeros, subnormals, infinities and NaN.  Prints the number of differences.
#include <cmath>
#include <cstdio>
#include <random>

#include "emcg_exp.h"

int main() {
  std::mt19937_64 g(5);
  long bad = 0;
  auto one = [&](double x) {
    const float a = (float)x, b = emcg::toFloat(x);
    bad += std::isnan(a) ? !std::isnan(b) : emcg::fbits(a) != emcg::fbits(b);
  };
  auto back = [&](float v) {
    const double a = (double)v, b = emcg::toDouble(v);
    bad += std::isnan(a) ? !std::isnan(b) : emcg::dbits(a) != emcg::dbits(b);
  };
  for (int i = 0; i < 4000000; i++) {
    uint64_t b = g();
    if (i & 1) // exponents from below the smallest subnormal float to above the largest
      b = (b & 0x800fffffffffffffull) | ((uint64_t)(860 + g() % 340) << 52);
    if (i % 5 == 0)
      b = (b & ~0x1fffffffull) | (0x0fffffffull + g() % 3);
    one(emcg::bitsd(b));
    back(emcg::bitsf((uint32_t)g()));
  }
  for (uint32_t e = 0; e < 256; e++)
    for (uint32_t m : {0u, 1u, 0x7ffffeu, 0x7fffffu})
      for (uint32_t s : {0u, 0x80000000u})
        back(emcg::bitsf(s | e << 23 | m));
  for (uint64_t e = 0; e < 2048; e++)
    for (uint64_t m : {0ull, 1ull, 0x10000000ull, 0xfffffefffffffull, 0xfffffffffffffull})
      for (uint64_t s : {0ull, 1ull << 63})
        one(emcg::bitsd(s | e << 52 | m));
  std::printf("%ld\n", bad);
  return 0;
}
