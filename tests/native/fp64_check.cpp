// emcg_fp64.h against the plain expressions it stands for: prints the number of
// disagreements of belowD and of fixedOf.
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
  std::printf("%ld %ld\n", badBelow, badFixed);
  return 0;
}
