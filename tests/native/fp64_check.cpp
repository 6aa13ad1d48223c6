// emcg_fp64.h against the plain expressions it stands for: prints the number of
// disagreements of the comparisons and of fixedOf, and the largest errors of rsqrtStep and
// rcpStep in units of the last place, from approximations of 20 fraction bits within
// 2^-20 of the value (the instructions' form).
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "emcg_fp64.h"

int main() {
  using namespace emcg;
  std::mt19937_64 g(3);
  std::vector<double> v = {0.0, -0.0, 5e-324, -5e-324, 1e-310, -1e-310, 1.0, -1.0, NAN, -NAN,
                           INFINITY, -INFINITY, 1.7e308, -1.7e308, 2.2250738585072014e-308};
  for (int i = 0; i < 200; i++)
    v.push_back(bitsd(g()));
  long badBelow = 0, badFixed = 0;
  for (double a : v)
    for (double b : v)
      if (b >= 0 && !std::signbit(b))
        badBelow += belowD(a, b) != (a < b);
  for (double a : v)
    badBelow += (negativeD(a) != (a < 0)) + (notPositiveD(a) != (a <= 0));
  std::uniform_real_distribution<double> e(-40, 33);
  for (double q : v) {
    uint64_t f = 0;
    badFixed += fixedOf(q, f) != (q >= 0 && q < 0x1p30 && !std::signbit(q));
  }
  for (int i = 0; i < 1000000; i++) {
    const double q = i < 1000 ? i / 8.0 : std::exp2(e(g));
    uint64_t f = 0;
    const bool in = fixedOf(q, f);
    badFixed += in != (q < 0x1p30) || (in && f != (uint64_t)std::floor(q * 0x1p20));
  }
  double worst[2] = {0, 0};
  std::uniform_real_distribution<double> x(-1000, 1000);
  for (int i = 0; i < 4000000; i++) {
    const double t = std::exp2(i & 1 ? x(g) : x(g) * 0.002);
    for (int k = 0; k < 2; k++) {
      const long double want = k ? 1.0L / (long double)t : 1.0L / std::sqrt((long double)t);
      // the 20-bit neighbour below or above
      const double y = bitsd((dbits((double)want) & ~0xffffffffull) + ((g() & 1) << 32));
      const double got = k ? rcpStep(t, y) : rsqrtStep(t, y);
      const double ulp = std::ldexp(1.0, std::ilogb((double)want) - 52);
      worst[k] = std::fmax(worst[k], (double)std::fabs(((long double)got - want) / ulp));
    }
  }
  std::printf("%ld %ld %.4f %.4f\n", badBelow, badFixed, worst[0], worst[1]);
  return 0;
}
