// emcg::canonicalBits and emcg::levelFast against the plain expressions they
// stand for, at the edges and on random arguments: prints the number of
// arguments where they differ.
#include <cmath>
#include <cstdio>
#include <random>

#include "emcg_draws.h"

static double canonical(uint64_t w) {
  const double r = (double)w * 0x1p-64;
  return r >= 1.0 ? 0x1.fffffffffffffp-1 : r;
}

int main() {
  std::mt19937_64 g(3);
  long bad = 0;
  auto word = [&](uint64_t w) { bad += emcg::dbits(canonical(w)) != emcg::dbits(emcg::canonicalBits(w)); };
  for (int s = 0; s < 64; s++)
    for (int64_t d = -3000; d <= 3000; d++)
      word(((uint64_t)1 << s) + (uint64_t)d);
  for (int i = 0; i < 4000000; i++) {
    const uint64_t w = g();
    word(w >> (i % 64));
    word((w >> (i % 53) & ~0x7ffull) | 0x400u); // ties
  }
  for (int nL : {1, 7, 1000, 3000})
    for (double maxE : {1.0, 3.0, 4.0, 0.7}) {
      const double dE = maxE / nL, inv = 1.0 / dE;
      auto level = [&](double E) { bad += emcg::levelExact(E, dE, nL) != emcg::levelFast(E, dE, inv, nL); };
      for (int k = 0; k <= nL + 3; k++) {
        double lo = k * dE, hi = lo;
        for (int u = 0; u < 40; u++) { // every energy around the level's bound
          level(lo);
          level(hi);
          lo = std::nextafter(lo, -INFINITY);
          hi = std::nextafter(hi, INFINITY);
        }
      }
      std::uniform_real_distribution<double> u(-0.1 * maxE, 1.5 * maxE);
      for (int i = 0; i < 300000; i++)
        level(u(g));
      for (double E : {0.0, -0.0, 5e-324, 1e-300, 1e30, 1e300, -1e300, (double)INFINITY,
                       -(double)INFINITY, (double)NAN, -(double)NAN, 2147483648.0 * dE,
                       4294967296.0 * dE})
        level(E);
    }
  std::printf("%ld\n", bad);
  return 0;
}
