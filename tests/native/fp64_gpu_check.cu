// emcg_fp64.cuh on the GPU: prints the number of approximations with bits below the
// 20th fraction bit, their largest relative error in 2^-20, the largest errors of
// rsqrtD, rcpD, sqrtD and divD in units of the last place, and the number of
// arguments at the ends of sqrtD's and divD's ranges where they are not the library's
// result or its neighbour, or outside them where they are not the library's.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "emcg_fp64.cuh"

using namespace emcg;

// o[0..5]: the approximations of 1 / sqrt(a) and 1 / a, then the four functions;
// o[6], o[7]: the library's root and quotient
__global__ void evaluate(int n, const double *__restrict__ a, const double *__restrict__ b,
                         double *__restrict__ o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  double y, z;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a[i]));
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(z) : "d"(a[i]));
  const double v[8] = {y, z, rsqrtD(a[i]), rcpD(a[i]), sqrtD(a[i]), divD(b[i], a[i]),
                       sqrt(a[i]), b[i] / a[i]};
  for (int k = 0; k < 8; k++)
    o[(size_t)k * n + i] = v[k];
}

static bool run(const std::vector<double> &a, const std::vector<double> &b,
                std::vector<double> &o) {
  const int n = (int)a.size();
  o.resize((size_t)8 * n);
  double *d = nullptr;
  if (cudaMalloc(&d, sizeof(double) * 10 * n) != cudaSuccess)
    return false;
  cudaMemcpy(d, a.data(), sizeof(double) * n, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b.data(), sizeof(double) * n, cudaMemcpyHostToDevice);
  evaluate<<<(n + 255) / 256, 256>>>(n, d, d + n, d + 2 * (size_t)n);
  cudaMemcpy(o.data(), d + 2 * (size_t)n, sizeof(double) * 8 * n, cudaMemcpyDeviceToHost);
  return cudaDeviceSynchronize() == cudaSuccess && cudaFree(d) == cudaSuccess;
}

int main() {
  std::mt19937_64 g(5);
  std::uniform_real_distribution<double> x(-499, 499), s(-2, 2);
  const int n = 1 << 19;
  std::vector<double> a(n), b(n), o;
  for (int i = 0; i < n; i++) {
    a[i] = std::exp2(i & 1 ? x(g) : s(g));
    b[i] = std::exp2(i & 1 ? x(g) : s(g)) * (g() & 1 ? 1 : -1);
  }
  if (!run(a, b, o))
    return 1;
  long low = 0;
  double approx = 0, worst[4] = {};
  for (int i = 0; i < n; i++) {
    const long double t = a[i], root = std::sqrt(t);
    const long double want[6] = {1 / root, 1 / t, 1 / root, 1 / t, root, (long double)b[i] / t};
    for (int k = 0; k < 6; k++) {
      const double v = o[(size_t)k * n + i];
      if (k < 2) {
        low += (dbits(v) & 0xffffffffu) != 0;
        approx = std::fmax(approx, (double)std::fabs(v / want[k] - 1) * 0x1p20);
      } else {
        const double ulp = std::ldexp(1.0, std::ilogb((double)want[k]) - 52);
        worst[k - 2] = std::fmax(worst[k - 2], (double)std::fabs((v - want[k]) / ulp));
      }
    }
  }
  // the ends of the ranges (normal numbers; 2^-500 to 2^500) and what lies outside
  const double ends[] = {0.0, -0.0, 5e-324, 1e-310, 2.2250738585072014e-308, -1.0, 1.0, 3.0,
                         0x1p-500, 0x1.fffffffffffffp-501, 0x1p500, 0x1.fffffffffffffp499,
                         0x1p501, 0x1p1023, 1.7976931348623157e308, INFINITY, -INFINITY, NAN};
  std::vector<double> ea, eb;
  for (double p : ends)
    for (double q : ends) {
      ea.push_back(p);
      eb.push_back(q);
    }
  if (!run(ea, eb, o))
    return 1;
  long edges = 0;
  const size_t m = ea.size();
  for (size_t i = 0; i < m; i++)
    for (int k = 4; k < 6; k++) {
      const double got = o[k * m + i], lib = o[(k + 2) * m + i];
      const double p = std::fabs(ea[i]), q = k == 4 ? 1.0 : std::fabs(eb[i]);
      const bool in = k == 4 ? std::isnormal(p) && ea[i] > 0
                             : p >= 0x1p-500 && p < 0x1p500 && q >= 0x1p-500 && q < 0x1p500;
      if (in)
        edges += dbits(got) - dbits(lib) + 1 > 2;
      else
        edges += dbits(got) != dbits(lib) && !(std::isnan(got) && std::isnan(lib));
    }
  std::printf("%ld %.4f %.4f %.4f %.4f %.4f %ld\n", low, approx, worst[0], worst[1], worst[2],
              worst[3], edges);
  return 0;
}
