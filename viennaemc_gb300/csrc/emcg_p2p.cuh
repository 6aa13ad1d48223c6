// Particle-particle Coulomb sums of the reference's FMM particle handlers
// (include/ParticleHandler/emcFMMParticleHandler.hpp,
// examples/bulkSimulationFMM/FMMBulkParticleHandler.hpp), evaluated directly on
// the GPU in place of scalFMM's fast multipole method.
//
// For every target i and every other particle j (and every periodic copy of
// the box), the pair term of FP2PRCutoff::NonMutualParticles
// (include/ParticleHandler/FMM/FP2PRCutoff.hpp:64-100):
//   d = x_i - x_j, 1/r^2 and 1/r; closer than the cutoff radius the separation
//   is rescaled to the cutoff and 1/r, 1/r^2 take the cutoff's values;
//   force_i += -q_i q_j d / r^3,   potential_i += q_j / r.
// These are the sums scalFMM leaves in its particle containers; the handlers
// multiply them by their Coulomb factor (ke / eps_r, with their sign).
//
// Layout: several targets per thread; the sources staged through shared memory
// in tiles that every thread of the block reads; when the targets alone give too
// few blocks, the tiles of a target block are split over a second grid
// dimension and the parts are added in order afterwards.  The pair arithmetic
// runs in the engine's precision, each tile's partial sums go to double
// accumulators.  The work is n^2 pair terms, bound by the FP32 (or FP64) pipes,
// not by memory:
// - float: 13 additions, multiplications and fused multiply-adds per pair, an
//   rsqrt and a minimum.  A thread's two targets are packed into register pairs,
//   so that the 13 issue as 6.5 packed instructions with the same results (add,
//   mul, fma .rn.f32x2), and the hardware's rsqrt is taken without the code
//   around it for subnormal arguments: a tile whose sums are not finite, as they
//   are with such an argument, is summed again with rsqrtf.  10.9 instructions
//   per pair instead of 19.5; the register reads of the packed instructions bound
//   it now (a loop of packed fma with distinct operands runs at 38 to 44 per clock
//   and SM, 64 with one operand): 1.31e12 -> 2.05e12 pairs/s at
//   32,768 charges, 1.73e12 -> 2.25e12 at 262,144.
// - double: an SM issues a double instruction of a warp every 16 clocks, so
//   their number counts: 18 per pair with 1 / r from the hardware's
//   approximation and one step of a third-order iteration, against 36 issue
//   slots with the division and the square root of the reference's order:
//   1.6e10 -> 3.1e10 pairs/s at 32,768 charges, 1.0e10 -> 2.9e10 at 5,001.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "emcg_fp64.cuh"
#include "emcg_host.h"

namespace emcg {

// threads per block, targets per thread and blocks per SM; a tile is the sources
// whose terms a target adds in T before the sum goes to double.  Float, 32,768
// targets (ms): 256 threads of 2 targets 0.589, 128 of 4 0.646, 64 of 8 0.826,
// 256 of 2 with 6 blocks per SM 0.606
template <class T> struct P2PShape;
template <> struct P2PShape<float> {
  static constexpr int kThreads = 256, kTargets = 2, kTile = 256, kBlocks = 5;
};
template <> struct P2PShape<double> {
  static constexpr int kThreads = 128, kTargets = 2, kTile = 128, kBlocks = 5;
};

// two floats in one register pair
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &a, float &b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ float lowOf(f32x2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ float rsqrtFast(float x) { // a subnormal x gives +inf
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The float pair term.  Closer than the cutoff the reference rescales d to the
// cutoff's length and takes 1/r and 1/r^2 at the cutoff, so the force factor
// d / r'^3 becomes d (1/r) (1/cut)^2 and the potential term q_j / cut: with c =
// min(1/r, 1/cut) the terms are d (1/r) c^2 q_j and c q_j on either side of the
// cutoff.  The target's charge and the force's sign are applied to the tile's
// sums, not to every pair.  (nx, ny, nz): the source's negated position.
__device__ __forceinline__ void pairTermF(float xi, float yi, float zi, float nx, float ny,
                                          float nz, float q, float invCut, float acc[4]) {
  const float dx = xi + nx, dy = yi + ny, dz = zi + nz;
  const float inv = rsqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz)));
  const float c = fminf(inv, invCut);
  const float w = inv * c * c * q;
  acc[0] = fmaf(dx, w, acc[0]);
  acc[1] = fmaf(dy, w, acc[1]);
  acc[2] = fmaf(dz, w, acc[2]);
  acc[3] = fmaf(c, q, acc[3]);
}
// the same for two targets; kSelf: the pair is left out for the target whose own
// source it is (self0, self1)
template <bool kSelf>
__device__ __forceinline__ void pairTermF2(f32x2 x, f32x2 y, f32x2 z, f32x2 nx, f32x2 ny, f32x2 nz,
                                           f32x2 q, float invCut, f32x2 acc[4],
                                           bool self0 = false, bool self1 = false) {
  const f32x2 dx = add2(x, nx), dy = add2(y, ny), dz = add2(z, nz);
  float r0, r1;
  unpack2(fma2(dx, dx, fma2(dy, dy, mul2(dz, dz))), r0, r1);
  if (kSelf) {
    float q0, q1;
    unpack2(q, q0, q1);
    r0 = self0 ? 1.f : r0;
    r1 = self1 ? 1.f : r1;
    q = pack2(self0 ? 0.f : q0, self1 ? 0.f : q1);
  }
  const float i0 = rsqrtFast(r0), i1 = rsqrtFast(r1);
  const f32x2 c = pack2(fminf(i0, invCut), fminf(i1, invCut));
  const f32x2 w = mul2(mul2(mul2(pack2(i0, i1), c), c), q);
  acc[0] = fma2(dx, w, acc[0]);
  acc[1] = fma2(dy, w, acc[1]);
  acc[2] = fma2(dz, w, acc[2]);
  acc[3] = fma2(c, q, acc[3]);
}

// The double pair term, the same form.  0, subnormal, infinite and NaN r^2 by the
// reference's 1 / r^2 and square root.
__device__ __forceinline__ void pairTermD(double xi, double yi, double zi, double nx, double ny,
                                          double nz, double q, double invCut, double acc[4]) {
  const double dx = xi + nx, dy = yi + ny, dz = zi + nz;
  const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
  const double inv = (uint32_t)__double2hiint(r2) - 0x00100000u < 0x7fe00000u ? rsqrtD(r2)
                                                                               : sqrt(1.0 / r2);
  // inv > invCut by the bit patterns (both >= 0; a NaN stays)
  const long long bi = __double_as_longlong(inv);
  const double c = bi > __double_as_longlong(invCut) && bi <= 0x7ff0000000000000ll ? invCut : inv;
  const double w = inv * c * c * q;
  acc[0] = fma(dx, w, acc[0]);
  acc[1] = fma(dy, w, acc[1]);
  acc[2] = fma(dz, w, acc[2]);
  acc[3] = fma(c, q, acc[3]);
}

// a staged source: position negated, charge; float: each value twice, as the
// packed terms take it
template <class T> struct Src4;
template <> struct __align__(16) Src4<float> { f32x2 x, y, z, q; };
template <> struct __align__(16) Src4<double> { double x, y, z, q; };

// How the sources are worked through: groups of `chunk` sources (the float sums'
// tiles start anew in each), `perChunk` tiles per group, `per` consecutive tiles
// per block of the second grid dimension.
struct P2PPlan {
  int64_t chunk;
  int perChunk, per, parts;
};

// Grid (target blocks, parts): each thread sums its part's sources (all periodic
// copies) for kTargets of the first nTgt particles and writes the partial sums
// part[part][4][nTgt]; p2pReduceKernel adds the parts in order.
template <class T>
__global__ void __launch_bounds__(P2PShape<T>::kThreads, P2PShape<T>::kBlocks)
    p2pKernel(const double *__restrict__ x, const double *__restrict__ y,
              const double *__restrict__ z, const double *__restrict__ q, int64_t n,
              int64_t nTgt, P2PPlan plan, T invCut, double box, int images,
              double *__restrict__ part) {
  constexpr int kThr = P2PShape<T>::kThreads, kTgt = P2PShape<T>::kTargets,
                kTile = P2PShape<T>::kTile;
  __shared__ Src4<T> tile[kTile];
  const int64_t block0 = (int64_t)blockIdx.x * kThr * kTgt, base = block0 + threadIdx.x;
  T xi[kTgt], yi[kTgt], zi[kTgt];
  __shared__ double sumF[kTgt * 4][kThr];
#pragma unroll
  for (int u = 0; u < kTgt; u++) {
    const int64_t i = base + (int64_t)u * kThr;
    const bool a = i < nTgt;
    xi[u] = a ? (T)x[i] : T(0);
    yi[u] = a ? (T)y[i] : T(0);
    zi[u] = a ? (T)z[i] : T(0);
#pragma unroll
    for (int v = 0; v < 4; v++)
      sumF[4 * u + v][threadIdx.x] = 0.;
  }
  const int tl0 = blockIdx.y * plan.per;
  for (int a = -images; a <= images; a++)
    for (int b = -images; b <= images; b++)
      for (int c = -images; c <= images; c++) {
        const bool central = a == 0 && b == 0 && c == 0;
        const double ox = a * box, oy = b * box, oz = c * box;
        for (int tl = tl0; tl < tl0 + plan.per; tl++) {
          const int ck = tl / plan.perChunk;
          const int64_t t0 = ck * plan.chunk + (int64_t)(tl - ck * plan.perChunk) * kTile;
          const int64_t t1 = min(min(n, (ck + 1) * plan.chunk), t0 + kTile);
          if (t0 >= t1) // past the group's end, or the last group's
            continue;
          const int cnt = (int)(t1 - t0);
          __syncthreads(); // the previous tile is consumed
          for (int k = threadIdx.x; k < cnt; k += kThr) {
            const int64_t j = t0 + k;
            const T nx = -(T)(x[j] + ox), ny = -(T)(y[j] + oy), nz = -(T)(z[j] + oz),
                    qj = (T)q[j];
            if constexpr (sizeof(T) == 4)
              tile[k] = Src4<T>{pack2(nx, nx), pack2(ny, ny), pack2(nz, nz), pack2(qj, qj)};
            else
              tile[k] = Src4<T>{nx, ny, nz, qj};
          }
          __syncthreads();
          // the self pair (central copy) is left out: where the tile holds some of
          // the block's targets its charge counts as 0 and its r^2 as 1
          const bool own = central && t0 < block0 + kThr * kTgt && block0 < t1;
          T acc[kTgt][4] = {};
          if constexpr (sizeof(T) == 4) {
            static_assert(kTgt == 2 || sizeof(T) != 4, "one packed pair per thread");
            const f32x2 px = pack2(xi[0], xi[1]), py = pack2(yi[0], yi[1]),
                        pz = pack2(zi[0], zi[1]);
            f32x2 pa[4] = {};
            if (!own) {
#pragma unroll 4
              for (int k = 0; k < cnt; k++) {
                const Src4<T> s = tile[k];
                pairTermF2<false>(px, py, pz, s.x, s.y, s.z, s.q, invCut, pa);
              }
            } else {
              const int self = (int)max(min(base - t0, (int64_t)1 << 30), -((int64_t)1 << 30));
#pragma unroll 2
              for (int k = 0; k < cnt; k++) {
                const Src4<T> s = tile[k];
                pairTermF2<true>(px, py, pz, s.x, s.y, s.z, s.q, invCut, pa, k == self,
                                 k == self + kThr);
              }
            }
            float all = 0.f;
#pragma unroll
            for (int v = 0; v < 4; v++) {
              unpack2(pa[v], acc[0][v], acc[1][v]);
              all += acc[0][v] + acc[1][v];
            }
            if (!isfinite(all)) { // a subnormal or zero r^2 (or an overflow): again, plainly
#pragma unroll
              for (int u = 0; u < kTgt; u++)
#pragma unroll
                for (int v = 0; v < 4; v++)
                  acc[u][v] = 0.f;
              for (int k = 0; k < cnt; k++) {
                const Src4<T> s = tile[k];
#pragma unroll
                for (int u = 0; u < kTgt; u++)
                  if (!(central && t0 + k == base + (int64_t)u * kThr))
                    pairTermF(xi[u], yi[u], zi[u], lowOf(s.x), lowOf(s.y), lowOf(s.z), lowOf(s.q),
                              invCut, acc[u]);
              }
            }
          } else if (!own) {
#pragma unroll 2
            for (int k = 0; k < cnt; k++) {
              const Src4<T> s = tile[k];
#pragma unroll
              for (int u = 0; u < kTgt; u++)
                pairTermD(xi[u], yi[u], zi[u], s.x, s.y, s.z, s.q, invCut, acc[u]);
            }
          } else {
            for (int k = 0; k < cnt; k++) {
              const Src4<T> s = tile[k];
#pragma unroll
              for (int u = 0; u < kTgt; u++)
                if (t0 + k != base + (int64_t)u * kThr)
                  pairTermD(xi[u], yi[u], zi[u], s.x, s.y, s.z, s.q, invCut, acc[u]);
            }
          }
          // the sums leave out the target's charge and the force's sign
#pragma unroll
          for (int u = 0; u < kTgt; u++)
#pragma unroll
            for (int v = 0; v < 4; v++)
              sumF[4 * u + v][threadIdx.x] += (double)acc[u][v];
        }
      }
  double *out = part + (size_t)blockIdx.y * 4 * nTgt;
#pragma unroll
  for (int u = 0; u < kTgt; u++) {
    const int64_t i = base + (int64_t)u * kThr;
    if (i < nTgt) {
      const double g = -(double)(T)q[i];
#pragma unroll
      for (int v = 0; v < 4; v++)
        out[(size_t)v * nTgt + i] = (v < 3 ? g : 1.) * sumF[4 * u + v][threadIdx.x];
    }
  }
}

// The parts' sums added in order (deterministic); quantity v of target i goes
// to out[v * stride + i].
static __global__ void __launch_bounds__(256)
    p2pReduceKernel(const double *__restrict__ part, int parts, int64_t n,
                    double *__restrict__ out, int64_t stride) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 4 * n)
    return;
  double s = 0.;
#pragma unroll 4
  for (int c = 0; c < parts; c++)
    s += part[(size_t)c * 4 * n + t];
  const int64_t v = t / n, i = t - v * n;
  out[v * stride + i] = s;
}

// The plan for nTgt targets and n sources: parts short enough for 16 blocks per
// SM, so that the last blocks leave few SMs idle.  Float: the groups of sources
// are as many as give 4 blocks of 512 targets per SM (they fix which terms are
// added in float), a part is some whole tiles (32,768 targets in 640 blocks of
// one group each, 4.2 per SM, left a sixth of the time).  Double: a part is a
// group, of at least 8 sources (1,000 targets: 500 blocks instead of 8).
template <class T> inline P2PPlan p2pPlan(int64_t nTgt, int64_t n, int sms) {
  using S = P2PShape<T>;
  P2PPlan p;
  const int64_t tBlocks = std::max<int64_t>(
      1, (nTgt + S::kThreads * S::kTargets - 1) / (S::kThreads * S::kTargets));
  int64_t chunks = sizeof(T) == 4
                       ? std::min<int64_t>((4LL * sms + tBlocks - 1) / tBlocks, (nTgt + 255) / 256)
                       : std::min<int64_t>(16LL * sms / tBlocks, (n + 7) / 8);
  chunks = std::max<int64_t>(1, std::min<int64_t>(chunks, 65535));
  p.chunk = std::max<int64_t>((n + chunks - 1) / chunks, 1);
  p.perChunk = (int)((p.chunk + S::kTile - 1) / S::kTile);
  const int64_t tiles = chunks * p.perChunk;
  const int64_t per = sizeof(T) == 4 ? tiles * tBlocks / (16LL * sms) : p.perChunk;
  p.per = (int)std::max<int64_t>(std::max<int64_t>(per, 1), (tiles + 65534) / 65535);
  p.parts = (int)((tiles + p.per - 1) / p.per);
  return p;
}

// Launch the sums over sources (x, y, z, q: n doubles each) for the first
// nTgt of them on stream st: part holds 4 * nTgt * plan.parts doubles, out
// receives force x, y, z and potential with the given stride.  inv_cutoff 0:
// no cutoff.
template <class T>
inline cudaError_t p2pLaunch(const double *x, const double *y, const double *z, const double *q,
                             int64_t n, int64_t nTgt, double invCutoff, double box, int images,
                             const P2PPlan &plan, double *part, double *out, int64_t stride,
                             cudaStream_t st) {
  using S = P2PShape<T>;
  if (nTgt <= 0)
    return cudaSuccess;
  const int64_t perBlock = S::kThreads * S::kTargets;
  const dim3 grid((unsigned)((nTgt + perBlock - 1) / perBlock), (unsigned)plan.parts);
  const double ic = invCutoff > 0 ? invCutoff : INFINITY; // no cutoff: no 1/r exceeds it
  p2pKernel<T><<<grid, S::kThreads, 0, st>>>(x, y, z, q, n, nTgt, plan, (T)ic, box, images, part);
  p2pReduceKernel<<<(unsigned)((4 * nTgt + 255) / 256), 256, 0, st>>>(part, plan.parts, nTgt, out,
                                                                      stride);
  return cudaGetLastError();
}

} // namespace emcg
