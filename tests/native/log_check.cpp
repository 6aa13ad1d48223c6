// Accuracy of emcg::logTab (the step kernel's log of its draws) against the
// host's extended-precision log: prints the largest error in units of the last
// place of the result over the draws' range, and whether 1 and the arguments
// handed to the library come out right.
#include <cmath>
#include <cstdio>
#include <random>

#include "emcg_log.h"

static double tab[emcg::kLogTab];

static double ulps(double x) {
  const double a = emcg::logTab(x, tab);
  const long double b = std::log((long double)x);
  return (double)(std::fabs((long double)a - b) /
                  ((long double)std::ldexp(1.0, std::ilogb((double)std::fabs(b)) - 52)));
}

int main() {
  for (int i = 0; i < emcg::kLogTab; i++)
    tab[i] = emcg::logTabEntry(i);
  double worst = 0, sum = 0, lib = 0;
  std::mt19937_64 g(11);
  std::uniform_real_distribution<double> u(1e-6, 1.0), s(std::log(1e-6), 0.0), o(-20.0, -0.1);
  const int n = 3000000;
  for (int i = 0; i < n; i++) {
    // uniform draws, small ones, and ones close to 1
    const double x = i % 3 == 0 ? u(g) : i % 3 == 1 ? std::exp(s(g)) : 1.0 - std::exp(o(g));
    if (x >= 1.0)
      continue;
    const double e = ulps(x);
    worst = std::fmax(worst, e);
    sum += e * e;
    const long double b = std::log((long double)x);
    lib = std::fmax(lib, (double)(std::fabs((long double)std::log(x) - b) /
                                  std::ldexp(1.0, std::ilogb((double)std::fabs(b)) - 52)));
  }
  // interval bounds, from below and above
  for (int j = 0; j <= emcg::kLogIntervals; j++)
    for (int k = 0; k < 20; k++) {
      const double a = std::ldexp(
          emcg::bitsd((uint64_t)(0x3fe60000u + (uint32_t)j * 0x2000u) << 32), -k);
      for (double x : {a, std::nextafter(a, 0.0), std::nextafter(a, 2.0)})
        if (x != 1.0 && x < 2.0)
          worst = std::fmax(worst, ulps(x));
    }
  const bool specials = emcg::logTab(1.0, tab) == 0.0 && std::isinf(emcg::logTab(0.0, tab)) &&
                        std::isnan(emcg::logTab(-1.0, tab)) && std::isnan(emcg::logTab(NAN, tab)) &&
                        emcg::logTab(3.0, tab) == std::log(3.0) &&
                        emcg::logTab(1e-300, tab) == std::log(1e-300);
  std::printf("%.4f %.4f %.4f %d\n", worst, std::sqrt(sum / n), lib, specials ? 1 : 0);
  return 0;
}
