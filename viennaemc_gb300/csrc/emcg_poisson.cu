// Grid Poisson solver of the device engine: double-precision Newton / defect
// correction around geometric multigrid V-cycles (see emcg_poisson.cuh).
#include <algorithm>
#include <array>
#include <atomic>
#include <map>
#include <cmath>
#include <cstring>
#include <vector>

#include <cooperative_groups.h>

#include "emcg_common.cuh"
#include "emcg_exp.h"
#include "emcg_host.h"
#include "emcg_poisson.cuh"

namespace emcg {

namespace cg = cooperative_groups;

namespace {

constexpr int kBlock = 256;
constexpr double kMaxNewtonStep = 2.0; // thermal voltages per iteration

__device__ __forceinline__ void atomicMaxPos(double *addr, double v) {
  // non-negative doubles order like their bit patterns
  atomicMax(reinterpret_cast<unsigned long long *>(addr), (unsigned long long)__double_as_longlong(v));
}

__device__ __forceinline__ double blockMax(double v) {
  __shared__ double sh[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0)
    sh[w] = v;
  __syncthreads();
  if (w == 0) {
    v = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  }
  return v; // valid in thread 0
}

// Gauss-Seidel update s / (diagonal) as s times the diagonal's reciprocal,
// which the cluster solve's sweeps form once: the float smoother's by the
// hardware's approximation (its error is far below the float multigrid's own
// 1e-7).  The double smoother's quotients are a unit in the last place off where the
// product rounds twice; they are corrections only, and with exact quotients the
// potential's error against 64-bit Newton with conjugate gradients is the same in
// every digit shown (five grids, 1.3e-13 to 4.9e-11), in 5 to 12 % more time.
__device__ __forceinline__ float mgRcp(float den) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(den));
  return r;
}
__device__ __forceinline__ double mgRcp(double den) { return 1.0 / den; }

__global__ void resetBCKernel(double *pot, const uint8_t *mask, const double *val, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && mask[i])
    pot[i] = val[i];
}

// x is finite (neither an infinity nor a NaN), by its exponent bits: no
// double-precision instruction
__device__ __forceinline__ bool finiteBits(double x) {
  return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000;
}

// max of two non-negative doubles (+0 to +inf; a NaN ranks above all) by
// their bit patterns, which order like the values: integer instructions only
__device__ __forceinline__ unsigned long long bitsMax(unsigned long long a, unsigned long long b) {
  return a > b ? a : b;
}
__device__ __forceinline__ double dmaxPos(double a, double b) {
  return __longlong_as_double(
      (long long)bitsMax((unsigned long long)__double_as_longlong(a),
                         (unsigned long long)__double_as_longlong(b)));
}

// a > 0, and a < b, for non-negative a and b, without a double-precision instruction
__device__ __forceinline__ bool bitsPositive(double a) { return __double_as_longlong(a) > 0; }
__device__ __forceinline__ bool bitsBelow(double a, double b) {
  return __double_as_longlong(a) < __double_as_longlong(b);
}

// F(phi) at node i = (x, y) of the reference equation (the SOR fixed point
// of emcSORSolver.hpp:131-197 times the FV area), with p = exp(-phi) and n
// (the concentration, or exp(phi) at equilibrium).  Both solve paths call this
// one function, so they see the same values to the last bit.  Written for the
// GPU's narrow double-precision pipes: the table exp, the stencil as three
// fused multiply-adds, and the gate terms only where a gate contact is (their
// sums are zero elsewhere, and adding zero changes nothing).
struct NodeF {
  double F, p, n;
};
struct NodeIn { // what it reads: the potential at the node and beside it, the rest there
  double phi, w, e, s, nn, gs, gv, conc, C;
};
__device__ __forceinline__ NodeIn nodeLoad(const double *__restrict__ pot,
                                           const double *__restrict__ conc,
                                           const double *__restrict__ C,
                                           const double *__restrict__ gSum,
                                           const double *__restrict__ gV, int i, int x, int y,
                                           int nx, int ny) {
  NodeIn q;
  q.phi = pot[i];
  q.w = x > 0 ? pot[i - 1] : pot[i + 1];
  q.e = x < nx - 1 ? pot[i + 1] : pot[i - 1];
  q.s = y > 0 ? pot[i - nx] : pot[i + nx];
  q.nn = y < ny - 1 ? pot[i + nx] : pot[i - nx];
  q.gs = gSum[i];
  q.gv = gV[i];
  q.conc = conc ? conc[i] : 0.;
  q.C = C[i];
  return q;
}
__device__ __forceinline__ NodeF nodeResidual(const NodeIn &q, bool conc, double hF0, double hF1,
                                              double c2, double hP, const double *tab) {
  NodeF r;
  r.p = expTab(bitsd(dbits(q.phi) ^ 0x8000000000000000ull), tab);
  r.n = conc ? q.conc : expTab(q.phi, tab);
  double F = hF0 * (q.w + q.e);
  F = fma(hF1, q.s + q.nn, F);
  F = fma(c2, q.phi, F); // c2 = -2 (hF0 + hF1)
  F = fma(hP, (r.p - r.n) + q.C, F);
  if (((__double_as_longlong(q.gs) | __double_as_longlong(q.gv)) << 1) != 0)
    F += q.gv - q.gs * q.phi;
  r.F = F;
  return r;
}
// in the multigrid's type, and back
template <class MT> __device__ __forceinline__ MT mgOf(double x) {
  if constexpr (sizeof(MT) == 4)
    return toFloat(x);
  else
    return x;
}
__device__ __forceinline__ double doubleOf(float v) { return toDouble(v); }
__device__ __forceinline__ double doubleOf(double v) { return v; }

// F(phi) of the reference equation, the Jacobian's reaction density and the
// FV-scaled right-hand side of the correction equation on level 0.
template <class MT>
__global__ void nonlinResidualKernel(const double *__restrict__ pot, const double *__restrict__ conc,
                                     const double *__restrict__ C, const uint8_t *__restrict__ fixed,
                                     const double *__restrict__ gSum, const double *__restrict__ gV,
                                     int nx, int ny, double hF0, double hF1, double hP,
                                     MT *__restrict__ rhs, MT *__restrict__ rho, MT *__restrict__ d,
                                     double *__restrict__ stats, int withScale) {
  __shared__ double tab[kExpTab]; // 2^(j/256) for expTab
  for (int k = threadIdx.x; k < kExpTab; k += blockDim.x)
    tab[k] = exp2(k * (1.0 / kExpTab));
  __syncthreads();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  MT aF = 0;
  double sc = 0.;
  if (i < nx * ny) {
    d[i] = MT(0);
    if (fixed[i]) {
      rhs[i] = MT(0);
      rho[i] = MT(0);
    } else {
      int x = i % nx, y = i / nx;
      const NodeF q = nodeResidual(nodeLoad(pot, conc, C, gSum, gV, i, x, y, nx, ny),
                                   conc != nullptr, hF0, hF1, -2.0 * (hF0 + hF1), hP, tab);
      const double F = q.F, p = q.p, n = q.n;
      int bd = (x == 0 || x == nx - 1) + (y == 0 || y == ny - 1);
      // the FV scale (1, 1/2, 1/4) and the maxima in the multigrid's type:
      // exact scalings, and the maximum needs no more than float accuracy
      const MT fF = mgOf<MT>(F);
      rhs[i] = fF * (bd == 0 ? MT(1) : (bd == 1 ? MT(0.5) : MT(0.25)));
      rho[i] = mgOf<MT>(conc ? p : p + n);
      aF = fabs(fF);
      if (withScale)
        sc = hP * (fabs(C[i]) + n + p);
      // a NaN would vanish in the maxima (fmax drops it): a non-finite
      // residual or scale term counts as an infinite residual, which ends
      // the solve as not converged
      if (!finiteBits(F) || !finiteBits(sc) || !isfinite(fF))
        aF = INFINITY;
    }
  }
  double m1 = blockMax((double)aF);
  __syncthreads();
  double m2 = withScale ? blockMax(sc) : 0.;
  if (threadIdx.x == 0) {
    atomicMaxPos(&stats[0], m1);
    if (withScale)
      atomicMaxPos(&stats[1], m2);
  }
}

// 2^(j/256), j < 256, for expTab: the same values as the multi-launch
// residual kernel forms in its shared memory
__global__ void expTableKernel(double *tab) {
  const int k = threadIdx.x;
  if (k < kExpTab)
    tab[k] = exp2(k * (1.0 / kExpTab));
}

template <class MT>
__global__ void updatePotKernel(double *__restrict__ pot, const MT *__restrict__ d,
                                const uint8_t *__restrict__ fixed, int n, double *stats) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  MT a = 0;
  if (i < n && !fixed[i]) {
    // clamped in the correction's own type (the bound is exact in float)
    MT v = d[i];
    // the clamp would turn a NaN correction into -kMaxNewtonStep (fmax drops
    // NaN): a non-finite correction is passed on, so that the next residual
    // reports it
    if (isfinite(v))
      v = fmin(MT(kMaxNewtonStep), fmax(MT(-kMaxNewtonStep), v));
    pot[i] += doubleOf(v);
    a = isfinite(v) ? fabs(v) : MT(INFINITY);
  }
  double m = blockMax((double)a);
  if (threadIdx.x == 0)
    atomicMaxPos(&stats[2], m);
}

template <class MT> struct LevelK {
  int nx, ny;
  const MT *cw, *ce, *cs, *cn, *area, *diag0;
  const uint8_t *fixed;
  MT *d, *r, *rho;
};

// (the sums of the multigrid are written as fused multiply-adds in both solve
// paths, so that they round alike whatever the compiler would contract)
template <class MT>
__device__ __forceinline__ MT applyRow(const LevelK<MT> &L, int i, int x, int y, MT di) {
  MT s = fma(L.area[i], L.rho[i], L.diag0[i]) * di;
  if (x > 0)
    s = fma(-L.cw[i], L.d[i - 1], s);
  if (x < L.nx - 1)
    s = fma(-L.ce[i], L.d[i + 1], s);
  if (y > 0)
    s = fma(-L.cs[i], L.d[i - L.nx], s);
  if (y < L.ny - 1)
    s = fma(-L.cn[i], L.d[i + L.nx], s);
  return s;
}
// the Gauss-Seidel value of node i
template <class MT>
__device__ __forceinline__ MT sweepValue(const LevelK<MT> &L, int i, int x, int y) {
  MT s = L.r[i];
  if (x > 0)
    s = fma(L.cw[i], L.d[i - 1], s);
  if (x < L.nx - 1)
    s = fma(L.ce[i], L.d[i + 1], s);
  if (y > 0)
    s = fma(L.cs[i], L.d[i - L.nx], s);
  if (y < L.ny - 1)
    s = fma(L.cn[i], L.d[i + L.nx], s);
  return s * mgRcp(fma(L.area[i], L.rho[i], L.diag0[i]));
}

template <class MT> __global__ void smoothKernel(LevelK<MT> L, int color) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  // thread t handles the t-th node of the colour
  int half = (L.nx + 1) / 2;
  int y = t / half;
  if (y >= L.ny)
    return;
  int x = 2 * (t - y * half) + ((y + color) & 1);
  if (x >= L.nx)
    return;
  int i = y * L.nx + x;
  if (L.fixed[i])
    return;
  L.d[i] = sweepValue(L, i, x, y);
}

// coarse rhs = P^T (fine residual); coarse reaction by injection; coarse d = 0
template <class MT>
__global__ void restrictKernel(LevelK<MT> F, LevelK<MT> Cc, const int *rxIdx, const float *rxW,
                               const int *ryIdx, const float *ryW, const int *mapX,
                               const int *mapY) {
  int I = blockIdx.x * blockDim.x + threadIdx.x;
  if (I >= Cc.nx * Cc.ny)
    return;
  int X = I % Cc.nx, Y = I / Cc.nx;
  Cc.d[I] = MT(0);
  Cc.rho[I] = F.rho[mapY[Y] * F.nx + mapX[X]];
  if (Cc.fixed[I]) {
    Cc.r[I] = MT(0);
    return;
  }
  MT acc = MT(0);
  for (int b = 0; b < 3; b++) {
    MT wy = (MT)ryW[3 * Y + b];
    if (wy == MT(0))
      continue;
    int y = ryIdx[3 * Y + b];
    for (int a = 0; a < 3; a++) {
      MT wx = (MT)rxW[3 * X + a];
      if (wx == MT(0))
        continue;
      int x = rxIdx[3 * X + a];
      int i = y * F.nx + x;
      if (F.fixed[i])
        continue;
      acc = fma(wx * wy, F.r[i] - applyRow(F, i, x, y, F.d[i]), acc);
    }
  }
  Cc.r[I] = acc;
}

template <class MT>
__global__ void prolongKernel(LevelK<MT> F, LevelK<MT> Cc, const int *pxIdx, const float *pxW,
                              const int *pyIdx, const float *pyW) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= F.nx * F.ny || F.fixed[i])
    return;
  int x = i % F.nx, y = i / F.nx;
  int X0 = pxIdx[x], Y0 = pyIdx[y];
  MT wx = (MT)pxW[x], wy = (MT)pyW[y];
  MT v = wx * wy * Cc.d[Y0 * Cc.nx + X0];
  if (wx < MT(1))
    v = fma((MT(1) - wx) * wy, Cc.d[Y0 * Cc.nx + X0 + 1], v);
  if (wy < MT(1)) {
    v = fma(wx * (MT(1) - wy), Cc.d[(Y0 + 1) * Cc.nx + X0], v);
    if (wx < MT(1))
      v = fma((MT(1) - wx) * (MT(1) - wy), Cc.d[(Y0 + 1) * Cc.nx + X0 + 1], v);
  }
  F.d[i] = F.d[i] + v;
}

// coarsest level: red-black sweeps inside one block
template <class MT> __global__ void coarseSolveKernel(LevelK<MT> L, int sweeps) {
  const int n = L.nx * L.ny;
  for (int it = 0; it < sweeps; it++) {
    for (int color = 0; color < 2; color++) {
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        int x = i % L.nx, y = i / L.nx;
        if (((x + y) & 1) != color || L.fixed[i])
          continue;
        L.d[i] = sweepValue(L, i, x, y);
      }
      __syncthreads();
    }
  }
}

template <class MT> LevelK<MT> levelK(const MGLevel &l);
template <> LevelK<float> levelK<float>(const MGLevel &l) {
  return {l.nx, l.ny, l.cw, l.ce, l.cs, l.cn, l.area, l.diag0, l.fixed, l.d, l.r, l.rho};
}
template <> LevelK<double> levelK<double>(const MGLevel &l) {
  return {l.nx, l.ny, l.dcw, l.dce, l.dcs, l.dcn, l.darea, l.ddiag0, l.fixed, l.dd, l.dr, l.drho};
}

// ---------------------------------------------------------------------------
// The whole solve in one launch of one thread-block cluster.
//
// Device-engine grids hold at most a few 1e5 nodes and stay on chip, so the
// multi-launch solve is bound by launch and host-synchronisation latency (one
// V-cycle is ~90 dependent phases), not by bandwidth.  Here one cluster of up to
// 16 CTAs runs the Newton / defect-correction loop, every V-cycle and the
// convergence test, with everything a phase touches in shared memory:
//  - rows of each level are split over the CTAs in bands, aligned between
//    levels where the sizes allow (a CTA's coarse rows lie under its fine
//    rows); the correction d, right-hand side r, reaction rho and residual of
//    every level live in the owning CTA, neighbours' rows are read through
//    distributed shared memory; the double potential stays in global memory,
//    read and written only by the residual and update phases;
//  - the static coefficients are a per-node class index into a small table of
//    the level's distinct coefficient tuples; they and the transfer tables are
//    staged once per launch;
//  - levels with at most kSmallNodes nodes live whole in CTA 0, which runs the
//    coarse part of every V-cycle alone with block barriers (warp barriers on
//    levels of at most kWarpNodes, which warp 0 works alone), the coarsest
//    grid in the registers of one warp;
//  - rows in a CTA's own shared memory are addressed from the kernel's
//    shared-memory base, so their loads and stores are shared-memory
//    instructions rather than generic ones; the sweeps keep each thread's nodes
//    in registers (cSweepsHeld);
//  - phases over distributed levels are separated by cluster barriers
//    (release / acquire).
// Every phase evaluates the expressions of the corresponding multi-launch
// kernel on the same values, so both paths give the same potential.
// ---------------------------------------------------------------------------
constexpr int kClusterThreads = 512;
constexpr int kMaxCluster = 16;
constexpr int kSmallNodes = 4096;
// levels below the finest of at most this many nodes (all held by CTA 0) are
// worked by warp 0 alone, its phases ending in __syncwarp instead of a
// barrier of the whole CTA.  Measured on the 201 x 101 resistor: 64 nodes
// (8x5 and coarser) -0.3 %, 128 nodes +5 %, 512 nodes +31 % against none:
// one warp walks a larger level's nodes one after another.
constexpr int kWarpNodes = 64;
constexpr size_t kClusterSmemMax = 227 * 1024;

// q = t / d for 0 <= t and t * d < 2^32, by one wide multiply (m = ceil(2^32 / d))
struct FastDiv {
  unsigned long long m;
  __host__ void set(unsigned d) { m = ((1ull << 32) + d - 1) / d; }
  __device__ __forceinline__ int div(int t) const {
    return (int)(((unsigned long long)(unsigned)t * m) >> 32);
  }
};

template <class MT> struct CLevel {
  int nx, ny, small, rowsPer; // small: all rows in CTA 0; else rowsPer rows per CTA
  int nCls, ncx, ncy, warp;   // ncx, ncy: next level's size (0 on the coarsest);
                              // warp: worked by warp 0 of CTA 0 alone
  FastDiv byNx, byHalf, byRows; // nx, (nx + 1) / 2 and rowsPer
  // byte offsets in dynamic shared memory: this CTA's rows of d, r, rho, the
  // residual and the class index, the class table (8 MT per class) and the
  // transfer tables to the next level (prolongation index / weight per fine x
  // and y, restriction 3 per coarse index, injection map)
  unsigned offD, offR, offRho, offRes, offCls, offTab;
  unsigned offCo; // the coarse rows under the CTA's rows (cStageCoarse); 0: no room
  unsigned offPxI, offPxW, offPyI, offPyW, offRxI, offRxW, offRyI, offRyW, offMapX, offMapY;
  const uint8_t *cls; // global sources staged at launch
  const MT *tab;
  const int *rxIdx, *ryIdx, *pxIdx, *pyIdx, *mapX, *mapY;
  const float *rxW, *ryW, *pxW, *pyW;
};

template <class MT> struct CMG {
  int nLev, pre, post, coarseSweeps, firstSmall, vcycles;
  double twoCycleRel;
  unsigned offRed;
  CLevel<MT> L[16];
};

struct CCtx {
  char *const *base; // generic address of each rank's dynamic shared memory
  char *smem;        // this CTA's dynamic shared memory
  int rank;
};

template <class MT> struct Coef {
  MT cw, ce, cs, cn, area, diag0, fixed, pad;
};

template <class MT> __device__ __forceinline__ Coef<MT> loadCoef(const MT *K);
template <> __device__ __forceinline__ Coef<float> loadCoef<float>(const float *K) {
  const float4 a = reinterpret_cast<const float4 *>(K)[0];
  const float4 b = reinterpret_cast<const float4 *>(K)[1];
  return {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
}
template <> __device__ __forceinline__ Coef<double> loadCoef<double>(const double *K) {
  const double2 a = reinterpret_cast<const double2 *>(K)[0];
  const double2 b = reinterpret_cast<const double2 *>(K)[1];
  const double2 e = reinterpret_cast<const double2 *>(K)[2];
  const double2 f = reinterpret_cast<const double2 *>(K)[3];
  return {a.x, a.y, b.x, b.y, e.x, e.y, f.x, f.y};
}

// rows [r0, r1) of level L held by this CTA
template <class MT>
__device__ __forceinline__ void cOwnRows(const CCtx &c, const CLevel<MT> &L, int &r0, int &r1) {
  if (L.small) {
    r0 = 0;
    r1 = c.rank == 0 ? L.ny : 0;
  } else {
    r0 = min(L.ny, c.rank * L.rowsPer);
    r1 = min(L.ny, r0 + L.rowsPer);
  }
}

template <class T> __device__ __forceinline__ const T *cTab(const CCtx &c, unsigned off) {
  return reinterpret_cast<const T *>(c.smem + off);
}

template <class MT>
__device__ __forceinline__ Coef<MT> cCoef(const CCtx &c, const CLevel<MT> &L, uint8_t k) {
  return loadCoef<MT>(reinterpret_cast<const MT *>(c.smem + L.offTab) + 8 * k);
}

// end of a phase over level L: cluster barrier for a distributed level, block
// barrier for one held by CTA 0, warp barrier for one worked by warp 0
template <class MT> __device__ __forceinline__ void cSync(const CLevel<MT> &L) {
  if (L.warp)
    __syncwarp();
  else if (L.small)
    __syncthreads();
  else
    cg::this_cluster().sync();
}

// threads that take no part in a phase over level L (warp-level levels: all
// but warp 0), and the stride of the threads that do
template <class MT> __device__ __forceinline__ bool cIdle(const CLevel<MT> &L) {
  return L.warp && threadIdx.x >= 32;
}
template <class MT> __device__ __forceinline__ int cStride(const CLevel<MT> &L) {
  return L.warp ? 32 : (int)blockDim.x;
}

// row ly of the CTA's own rows of an array of level L
template <class T, class MT>
__device__ __forceinline__ T *cOwn(const CCtx &c, const CLevel<MT> &L, unsigned off, int ly) {
  return reinterpret_cast<T *>(c.smem + off) + (size_t)ly * L.nx;
}

// Several red-black sweeps over level L with each thread's nodes held in
// registers: a thread keeps the same nodes of each colour over the three sweeps,
// so their position, class, right-hand side and the diagonal's reciprocal are
// formed once, and a half sweep reads only the coefficients and the neighbours'
// corrections.  The arithmetic is sweepValue's.
//
// A phase costs its longest chain of dependent instructions and what the four
// warps of a scheduler issue in it, not its work: so a thread's nodes go through
// each stage side by side, without branches -- all their loads, then the sums,
// then the stores (see heldNeighbours) --, a warp without nodes keeps the barriers
// only, and only a neighbour in another CTA's rows goes through distributed shared
// memory.  Measured on the 201 x 101 resistor's solves (two Newton steps): 0.399 ms
// with a branch per node and neighbour, 0.402 without branches but with every
// warp taking part, 0.323 with the idle warps out of the way, 0.301 with two
// nodes per thread where two are enough and the neighbours' addresses held.  On
// 401 x 201 0.735 -> 0.613 ms.
//
// kSweepNodes: nodes of one colour per thread.
constexpr int kSweepNodes = 3;
template <class MT> struct Held {
  unsigned a;    // shared address of the node's correction; 0: no node
  unsigned s, n; // of the neighbours below and above; bit 0: in another CTA
  unsigned k;    // shared address of its coefficients
  MT r, inv;     // right-hand side, 1 / diagonal
};

__device__ __forceinline__ float ldsAt(unsigned a, float) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ double ldsAt(unsigned a, double) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void stsIf(unsigned a, bool on, float v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p st.shared.f32 [%0], %2;\n\t}" ::"r"(a),
               "r"((unsigned)on), "f"(v)
               : "memory");
}
__device__ __forceinline__ void stsIf(unsigned a, bool on, double v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p st.shared.f64 [%0], %2;\n\t}" ::"r"(a),
               "r"((unsigned)on), "d"(v)
               : "memory");
}
// on: the value at shared address a, else 0
__device__ __forceinline__ float ldsIf(unsigned a, bool on, float) {
  float v;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
               "@p ld.shared.f32 %0, [%1];\n\t}"
               : "=f"(v)
               : "r"(a), "r"((unsigned)on)
               : "memory");
  return v;
}
__device__ __forceinline__ double ldsIf(unsigned a, bool on, double) {
  double v;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\tmov.f64 %0, "
               "0d0000000000000000;\n\t@p ld.shared.f64 %0, [%1];\n\t}"
               : "=d"(v)
               : "r"(a), "r"((unsigned)on)
               : "memory");
  return v;
}
// the same where the address may be another CTA's (far: a shared::cluster address)
__device__ __forceinline__ float ldsFar(unsigned a, bool on, bool far, float) {
  float v;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %2, 0;\n\tsetp.ne.u32 q, %3, 0;\n\t"
               "mov.f32 %0, 0f00000000;\n\t@p ld.shared.f32 %0, [%1];\n\t"
               "@q ld.shared::cluster.f32 %0, [%1];\n\t}"
               : "=f"(v)
               : "r"(a), "r"((unsigned)(on && !far)), "r"((unsigned)(on && far))
               : "memory");
  return v;
}
__device__ __forceinline__ double ldsFar(unsigned a, bool on, bool far, double) {
  double v;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %2, 0;\n\tsetp.ne.u32 q, %3, 0;\n\t"
               "mov.f64 %0, 0d0000000000000000;\n\t@p ld.shared.f64 %0, [%1];\n\t"
               "@q ld.shared::cluster.f64 %0, [%1];\n\t}"
               : "=d"(v)
               : "r"(a), "r"((unsigned)(on && !far)), "r"((unsigned)(on && far))
               : "memory");
  return v;
}
__device__ __forceinline__ unsigned mapShared(unsigned a, int rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}

// A level's array in this CTA's rows and the row above and below them: shared
// addresses, the neighbours' rows mapped.
struct NearRows {
  unsigned base, below, above; // own rows; row r0 - 1; row r0 + rowsPer
};
template <bool kS, class MT>
__device__ __forceinline__ NearRows nearRows(const CCtx &c, const CLevel<MT> &L, unsigned off) {
  NearRows n;
  n.base = (unsigned)__cvta_generic_to_shared(c.smem) + off;
  n.below = n.above = n.base;
  if (!kS) {
    if (c.rank > 0)
      n.below = mapShared(n.base + (unsigned)((L.rowsPer - 1) * L.nx * sizeof(MT)), c.rank - 1);
    if (c.rank + 1 < (int)cg::this_cluster().num_blocks())
      n.above = mapShared(n.base, c.rank + 1);
  }
  return n;
}
// element x of local row ly, where on
template <bool kS, class MT>
__device__ __forceinline__ MT nearLoad(const CLevel<MT> &L, const NearRows &n, int ly, int x,
                                       bool on) {
  if (kS)
    return ldsIf(n.base + (unsigned)((ly * L.nx + x) * (int)sizeof(MT)), on, MT());
  const bool lo = ly < 0, hi = ly >= L.rowsPer;
  const unsigned row = lo ? n.below : hi ? n.above : n.base + (unsigned)(ly * L.nx * (int)sizeof(MT));
  return ldsFar(row + (unsigned)(x * (int)sizeof(MT)), on, lo || hi, MT());
}

// the corrections beside a thread's nodes: past a row's end the next row's or the
// padding, past the domain's edge the node's own, all with a zero coefficient
template <bool kS, int N, class MT>
__device__ __forceinline__ void heldNeighbours(const Held<MT> (&h)[N], MT (&d)[N][4]) {
#pragma unroll
  for (int j = 0; j < N; j++) {
    d[j][0] = ldsAt(h[j].a - (unsigned)sizeof(MT), MT());
    d[j][1] = ldsAt(h[j].a + (unsigned)sizeof(MT), MT());
    if (kS) {
      d[j][2] = ldsAt(h[j].s, MT());
      d[j][3] = ldsAt(h[j].n, MT());
    } else {
      d[j][2] = ldsFar(h[j].s & ~1u, true, h[j].s & 1u, MT());
      d[j][3] = ldsFar(h[j].n & ~1u, true, h[j].n & 1u, MT());
    }
  }
}
__device__ __forceinline__ void coefAt(unsigned a, float (&c)[4]) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ void coefAt(unsigned a, double (&c)[4]) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(c[0]), "=d"(c[1]) : "r"(a) : "memory");
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];"
               : "=d"(c[2]), "=d"(c[3])
               : "r"(a + 16u)
               : "memory");
}

// the nodes threadIdx.x + (j0 + j) * stride of a colour of this CTA's rows; an
// absent or Dirichlet node reads the level's first and stores nothing
template <bool kS, int N, class MT>
__device__ __forceinline__ void loadHeld(const CCtx &c, const CLevel<MT> &L, const NearRows &nd,
                                         int r0, int cnt, int j0, int colour, Held<MT> (&h)[N]) {
  const int half = (L.nx + 1) / 2, stride = cStride(L);
  const unsigned base = nd.base - L.offD, row = (unsigned)(L.nx * (int)sizeof(MT));
  int q[N];
#pragma unroll
  for (int j = 0; j < N; j++) {
    const int t = threadIdx.x + (j0 + j) * stride, u = t < cnt ? t : 0;
    const int ly = L.byHalf.div(u), y = r0 + ly, x = 2 * (u - ly * half) + ((y + colour) & 1);
    const bool on = t < cnt && x < L.nx;
    const int i = on ? ly * L.nx + x : 0;
    h[j].a = nd.base + (unsigned)(i * (int)sizeof(MT));
    q[j] = *reinterpret_cast<const uint8_t *>(c.smem + L.offCls + i);
    h[j].s = on && y > 0 ? h[j].a - row : h[j].a;
    h[j].n = on && y < L.ny - 1 ? h[j].a + row : h[j].a;
    if (!kS) {
      if (on && y > 0 && ly == 0)
        h[j].s = (nd.below + (unsigned)(x * (int)sizeof(MT))) | 1u;
      if (on && y < L.ny - 1 && ly + 1 == L.rowsPer)
        h[j].n = (nd.above + (unsigned)(x * (int)sizeof(MT))) | 1u;
    }
    h[j].k = on ? 1u : 0u;
  }
  MT e[N][4];
#pragma unroll
  for (int j = 0; j < N; j++) {
    const unsigned k = base + L.offTab + (unsigned)(8 * q[j] * (int)sizeof(MT));
    h[j].r = ldsAt(h[j].a + (L.offR - L.offD), MT());
    h[j].inv = ldsAt(h[j].a + (L.offRho - L.offD), MT());
    coefAt(k + 4u * (unsigned)sizeof(MT), e[j]); // area, diagonal, fixed
    q[j] = (int)h[j].k;
    h[j].k = k;
  }
#pragma unroll
  for (int j = 0; j < N; j++)
    h[j].inv = q[j] && e[j][2] == MT(0) ? mgRcp(fma(e[j][0], h[j].inv, e[j][1])) : MT(0);
}

// a half sweep over nodes of a colour
template <bool kS, int N, class MT>
__device__ __forceinline__ void cHalfSweep(const CCtx &c, const CLevel<MT> &L, const NearRows &nd,
                                           int r0, const Held<MT> (&h)[N]) {
  MT f[N][4], d[N][4];
#pragma unroll
  for (int j = 0; j < N; j++)
    coefAt(h[j].k, f[j]);
  heldNeighbours<kS>(h, d);
#pragma unroll
  for (int j = 0; j < N; j++) {
    MT s = h[j].r;
#pragma unroll
    for (int q = 0; q < 4; q++)
      s = fma(f[j][q], d[j][q], s);
    stsIf(h[j].a, h[j].inv != MT(0), s * h[j].inv);
  }
}

// residual r - A d of the correction equation at nodes of a colour, as
// restrictKernel evaluates it (the Dirichlet nodes' zeros are written once, at
// the start of the launch)
template <bool kS, int N, class MT>
__device__ __forceinline__ void cResidualHeld(const CCtx &c, const CLevel<MT> &L,
                                              const NearRows &nd, int r0,
                                              const Held<MT> (&h)[N]) {
  MT f[N][4], e[N][4], d[N][4], rho[N], o[N];
#pragma unroll
  for (int j = 0; j < N; j++) {
    coefAt(h[j].k, f[j]);
    coefAt(h[j].k + 4u * (unsigned)sizeof(MT), e[j]); // area, diagonal, fixed
    rho[j] = ldsAt(h[j].a + (L.offRho - L.offD), MT());
    o[j] = ldsAt(h[j].a, MT());
  }
  heldNeighbours<kS>(h, d);
#pragma unroll
  for (int j = 0; j < N; j++) {
    MT s = fma(e[j][0], rho[j], e[j][1]) * o[j];
#pragma unroll
    for (int q = 0; q < 4; q++)
      s = fma(-f[j][q], d[j][q], s);
    stsIf(h[j].a + (L.offRes - L.offD), h[j].inv != MT(0), h[j].r - s);
  }
}

template <bool kS, int N, class MT>
__device__ __forceinline__ void cSweepsHeld(const CCtx &c, const CLevel<MT> &L, int r0, int cnt,
                                            int sweeps, int first, bool residual) {
  const NearRows nd = nearRows<kS>(c, L, L.offD);
  Held<MT> h[2][N];
  loadHeld<kS>(c, L, nd, r0, cnt, 0, 0, h[0]);
  loadHeld<kS>(c, L, nd, r0, cnt, 0, 1, h[1]);
  for (int s = 0; s < sweeps; s++) {
    if (first == 0) {
      cHalfSweep<kS>(c, L, nd, r0, h[0]);
      cSync(L);
      cHalfSweep<kS>(c, L, nd, r0, h[1]);
      cSync(L);
    } else {
      cHalfSweep<kS>(c, L, nd, r0, h[1]);
      cSync(L);
      cHalfSweep<kS>(c, L, nd, r0, h[0]);
      cSync(L);
    }
  }
  if (residual) {
    cResidualHeld<kS>(c, L, nd, r0, h[0]);
    cResidualHeld<kS>(c, L, nd, r0, h[1]);
    cSync(L);
  }
}

// the same for bands of more nodes than a thread holds, kBatchNodes at a time
constexpr int kBatchNodes = 4;
template <bool kS, class MT>
__device__ __forceinline__ void cSweepsBatch(const CCtx &c, const CLevel<MT> &L, int r0, int cnt,
                                             int sweeps, int first, bool residual) {
  const NearRows nd = nearRows<kS>(c, L, L.offD);
  const int per = (cnt + cStride(L) - 1) / cStride(L);
  for (int s = 0; s < 2 * sweeps + (residual ? 1 : 0); s++) {
    const bool res = s == 2 * sweeps;
    for (int k = 0; k < (res ? 2 : 1); k++)
      for (int j0 = 0; j0 < per; j0 += kBatchNodes) {
        Held<MT> h[kBatchNodes];
        loadHeld<kS>(c, L, nd, r0, cnt, j0, res ? k : (first + s) & 1, h);
        if (res)
          cResidualHeld<kS>(c, L, nd, r0, h);
        else
          cHalfSweep<kS>(c, L, nd, r0, h);
      }
    cSync(L);
  }
}

// Sweeps over a band of more rows than cSweepsHeld takes, held all the same: a
// thread keeps one column's nodes of either colour in every G-th row, so that their
// addresses are the first's plus multiples of a constant and a node costs two
// registers and a byte (right-hand side, reciprocal diagonal, class).  An even G
// keeps the colour's column.  kColNodes: rows of a thread at most.
// Measured on 401 x 201 in 16 CTAs (13 rows each), where every half sweep formed those
// nodes' constants anew before (cSweepsBatch): solve 0.566 -> 0.536 ms, two rows side by
// side (four: 0.541, by the registers); the 801 x 401 solve, whose tail it is, 1.815 ->
// 1.748.  Nine or ten rows a thread spill: 0.566; 17 rows (12 CTAs) stay with the other.
constexpr int kColNodes = 8;
// G of a level of nx columns in bands of rows: the threads' columns, an even number;
// 0: the column does not fit
__host__ __device__ constexpr int columnGroups(int nx, int rows) {
  const int G = kClusterThreads / ((nx + 1) / 2) & ~1;
  return rows <= kColNodes * G ? G : 0;
}
template <class MT> struct ColumnNodes {
  unsigned a0;                     // shared address of the first row's correction
  MT r[kColNodes], inv[kColNodes]; // inv 0: no node or a Dirichlet one
  unsigned cls[kColNodes / 4];     // four classes in each
};
struct Column {
  int g, G, R;            // first row, rows apart, the band's rows
  unsigned row;           // bytes of a row
  unsigned tab;           // the class table
  unsigned toS, toN;      // from the first and the last row to their outer neighbours, where
  bool below, above;      // another CTA has them
};
// d's address in row j of the column; rows past the band are its last
__device__ __forceinline__ unsigned columnAt(const Column &q, unsigned a0, int j, int &ly) {
  ly = min(q.g + j * q.G, q.R - 1);
  return a0 + (unsigned)(ly - q.g) * q.row;
}
template <bool kRes, class MT>
__device__ __forceinline__ void cColumnRows(const CLevel<MT> &L, const Column &q,
                                            const ColumnNodes<MT> &h) {
  constexpr int U = 2; // rows side by side (kColNodes is a multiple)
#pragma unroll
  for (int j0 = 0; j0 < kColNodes; j0 += U) {
    if (j0 * q.G >= q.R)
      break;
    MT f[U][4], d[U][4], e[U][4], rho[U], o[U];
    unsigned a[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      int ly;
      a[u] = columnAt(q, h.a0, j0 + u, ly);
      const unsigned k = q.tab + (h.cls[(j0 + u) / 4] >> 8 * ((j0 + u) & 3) & 0xffu) *
                                     (unsigned)(8 * sizeof(MT));
      coefAt(k, f[u]);
      if (kRes) {
        coefAt(k + 4u * (unsigned)sizeof(MT), e[u]); // area, diagonal, fixed
        rho[u] = ldsAt(a[u] + (L.offRho - L.offD), MT());
        o[u] = ldsAt(a[u], MT());
      }
      d[u][0] = ldsAt(a[u] - (unsigned)sizeof(MT), MT());
      d[u][1] = ldsAt(a[u] + (unsigned)sizeof(MT), MT());
      // beyond the domain's edge the node's own, with a zero coefficient
      const bool s = ly == 0, n = ly == q.R - 1;
      d[u][2] = ldsFar(a[u] + (s ? q.toS : 0u - q.row), true, s && q.below, MT());
      d[u][3] = ldsFar(a[u] + (n ? q.toN : q.row), true, n && q.above, MT());
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      MT s = kRes ? fma(e[u][0], rho[u], e[u][1]) * o[u] : h.r[j0 + u];
#pragma unroll
      for (int i = 0; i < 4; i++)
        s = fma(kRes ? -f[u][i] : f[u][i], d[u][i], s);
      stsIf(a[u] + (kRes ? L.offRes - L.offD : 0u), h.inv[j0 + u] != MT(0),
            kRes ? h.r[j0 + u] - s : s * h.inv[j0 + u]);
    }
  }
}
template <class MT>
__device__ __forceinline__ void columnLoad(const CCtx &c, const CLevel<MT> &L, const NearRows &nd,
                                           int r0, const Column &q, bool mine, int kx, int colour,
                                           ColumnNodes<MT> &h) {
  const int x = 2 * kx + ((r0 + q.g + colour) & 1);
  const bool on = mine && x < L.nx;
  h.a0 = nd.base + (unsigned)((q.g * L.nx + (on ? x : 0)) * (int)sizeof(MT));
#pragma unroll
  for (int j = 0; j < kColNodes; j++) {
    if (j % 4 == 0)
      h.cls[j / 4] = 0;
    h.r[j] = h.inv[j] = MT(0);
  }
#pragma unroll
  for (int j = 0; j < kColNodes; j++) {
    if (j * q.G >= q.R)
      break;
    int ly;
    const unsigned a = columnAt(q, h.a0, j, ly);
    const unsigned cls =
        *reinterpret_cast<const uint8_t *>(c.smem + (int)L.offCls + ly * L.nx + (on ? x : 0));
    MT e[4];
    coefAt(q.tab + (8 * cls + 4) * (unsigned)sizeof(MT), e);
    h.cls[j / 4] |= cls << 8 * (j & 3);
    h.r[j] = ldsAt(a + (L.offR - L.offD), MT());
    if (on && q.g + j * q.G < q.R && e[2] == MT(0))
      h.inv[j] = mgRcp(fma(e[0], ldsAt(a + (L.offRho - L.offD), MT()), e[1]));
  }
}
template <class MT>
__device__ __forceinline__ void cSweepsColumn(const CCtx &c, const CLevel<MT> &L, int r0, int R,
                                              int G, int sweeps, int first, bool residual) {
  const NearRows nd = nearRows<false>(c, L, L.offD);
  const int half = (L.nx + 1) / 2, g = L.byHalf.div(threadIdx.x);
  const bool mine = g < min(G, R);
  const int kx = mine ? (int)threadIdx.x - g * half : 0;
  Column q;
  q.g = mine ? g : 0;
  q.G = G;
  q.R = R;
  q.row = (unsigned)(L.nx * (int)sizeof(MT));
  q.tab = nd.base - L.offD + L.offTab;
  q.below = r0 > 0;
  q.above = r0 + R < L.ny;
  q.toS = q.below ? nd.below - nd.base : 0u;
  q.toN = q.above ? nd.above - (nd.base + (unsigned)(R - 1) * q.row) : 0u;
  ColumnNodes<MT> h[2];
  columnLoad(c, L, nd, r0, q, mine, kx, first, h[0]);
  columnLoad(c, L, nd, r0, q, mine, kx, first ^ 1, h[1]);
#pragma unroll 1
  for (int s = 0; s < sweeps; s++) {
    cColumnRows<false>(L, q, h[0]);
    cSync(L);
    cColumnRows<false>(L, q, h[1]);
    cSync(L);
  }
  if (residual) {
    cColumnRows<true>(L, q, h[0]);
    cColumnRows<true>(L, q, h[1]);
    cSync(L);
  }
}

// `sweeps` red-black sweeps over level L, colour `first` first, then (residual)
// the residual of the correction equation; every CTA passes the same
// 2 * sweeps (+ 1) barriers whichever form its rows take
template <bool kCol, class MT>
__device__ void cSmoothSweeps(const CCtx &c, const CLevel<MT> &Lr, int sweeps, int first,
                              bool residual = false) {
  const CLevel<MT> L = Lr;
  if (cIdle(L))
    return;
  int r0, r1;
  cOwnRows(c, L, r0, r1);
  const int cnt = (L.nx + 1) / 2 * (r1 - r0), stride = cStride(L);
  // nodes of a colour of this warp's first thread: a warp without any only keeps
  // the barriers (four warps share a scheduler, so what they issue in vain
  // delays the others)
  const int mine = (cnt - (int)(threadIdx.x & ~31u) + stride - 1) / stride;
  if (mine <= 0) {
    for (int s = 0; s < 2 * sweeps + (residual ? 1 : 0); s++)
      cSync(L);
  } else if (cnt <= kSweepNodes * stride) {
    if (L.small && mine == 1)
      cSweepsHeld<true, 1>(c, L, r0, cnt, sweeps, first, residual);
    else if (L.small && mine == 2)
      cSweepsHeld<true, 2>(c, L, r0, cnt, sweeps, first, residual);
    else if (L.small)
      cSweepsHeld<true, kSweepNodes>(c, L, r0, cnt, sweeps, first, residual);
    else if (mine == 1)
      cSweepsHeld<false, 1>(c, L, r0, cnt, sweeps, first, residual);
    else if (mine == 2)
      cSweepsHeld<false, 2>(c, L, r0, cnt, sweeps, first, residual);
    else
      cSweepsHeld<false, kSweepNodes>(c, L, r0, cnt, sweeps, first, residual);
  } else if (L.small) {
    cSweepsBatch<true>(c, L, r0, cnt, sweeps, first, residual);
  } else {
    if constexpr (kCol) {
      if (const int G = columnGroups(L.nx, L.rowsPer); G > 0) {
        cSweepsColumn(c, L, r0, r1 - r0, G, sweeps, first, residual);
        return;
      }
    }
    cSweepsBatch<false>(c, L, r0, cnt, sweeps, first, residual);
  }
}

// coarse rows whose injection row mapY[Y] this CTA holds: [Y0, Y1)
template <class MT>
__device__ __forceinline__ void cRestrictRows(const CCtx &c, const CLevel<MT> &F,
                                              const CLevel<MT> &Cc, int &Y0, int &Y1) {
  int r0, r1;
  cOwnRows(c, F, r0, r1);
  if (r0 >= r1) {
    Y0 = Y1 = 0;
    return;
  }
  if (F.ny <= 3) { // not coarsened along y: identity map
    Y0 = r0;
    Y1 = r1;
    return;
  }
  Y0 = (r0 + 1) / 2;
  Y1 = r1 == F.ny ? Cc.ny : min(Cc.ny, (r1 + 1) / 2);
}

// row Y of an array of the coarse level, wherever it lives
template <bool kS, class MT>
__device__ __forceinline__ char *cCoarseRow(const CCtx &c, const CLevel<MT> &Cc, int Y) {
  // (without the array's offset: one owner for the row's arrays)
  if (kS)
    return c.smem + (size_t)Y * Cc.nx * sizeof(MT);
  if (Cc.small)
    return (c.rank == 0 ? c.smem : c.base[0]) + (size_t)Y * Cc.nx * sizeof(MT);
  const int owner = Cc.byRows.div(Y);
  return (owner == c.rank ? c.smem : c.base[owner]) +
         (size_t)(Y - owner * Cc.rowsPer) * Cc.nx * sizeof(MT);
}

// coarse right-hand side P^T (fine residual), reaction by injection, d = 0; a
// coarse node is a Dirichlet node where the fine node under it is
// (U: coarse nodes of a thread side by side)
template <bool kS, int U, class MT>
__device__ __forceinline__ void cRestrictT(const CCtx &c, const CLevel<MT> &F,
                                           const CLevel<MT> &Cc) {
  int Y0, Y1, r0, r1;
  cRestrictRows(c, F, Cc, Y0, Y1);
  cOwnRows(c, F, r0, r1);
  const int cnt = Cc.nx * (Y1 - Y0), stride = cStride(F);
  const NearRows nr = nearRows<kS>(c, F, F.offRes);
  for (int t0 = threadIdx.x; t0 < cnt; t0 += U * stride) {
    int X[U], Y[U], xm[U], lym[U], xs[U][3], lys[U][3];
    MT wx[U][3], wy[U][3], rho[U], fixed[U], v[U][3][3];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int t = t0 + u * stride < cnt ? t0 + u * stride : t0;
      const int q = Cc.byNx.div(t);
      Y[u] = Y0 + q;
      X[u] = t - q * Cc.nx;
      xm[u] = cTab<int>(c, F.offMapX)[X[u]];
      lym[u] = cTab<int>(c, F.offMapY)[Y[u]] - r0;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        wx[u][k] = (MT)cTab<float>(c, F.offRxW)[3 * X[u] + k];
        wy[u][k] = (MT)cTab<float>(c, F.offRyW)[3 * Y[u] + k];
        xs[u][k] = cTab<int>(c, F.offRxI)[3 * X[u] + k];
        lys[u][k] = cTab<int>(c, F.offRyI)[3 * Y[u] + k] - r0;
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = lym[u] * F.nx + xm[u];
      const int q = *reinterpret_cast<const uint8_t *>(c.smem + F.offCls + i);
      rho[u] = reinterpret_cast<const MT *>(c.smem + F.offRho)[i];
      fixed[u] = reinterpret_cast<const MT *>(c.smem + F.offTab)[8 * q + 6];
#pragma unroll
      for (int b = 0; b < 3; b++)
#pragma unroll
        for (int a = 0; a < 3; a++) // a zero weight reads nothing (its row may be far)
          v[u][b][a] = nearLoad<kS>(F, nr, lys[u][b], xs[u][a],
                                    wx[u][a] != MT(0) && wy[u][b] != MT(0));
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      MT acc = MT(0);
#pragma unroll
      for (int b = 0; b < 3; b++)
#pragma unroll
        for (int a = 0; a < 3; a++)
          acc = fma(wx[u][a] * wy[u][b], v[u][b][a], acc);
      if (fixed[u] != MT(0))
        acc = MT(0);
      if (t0 + u * stride < cnt) {
        char *row = cCoarseRow<kS>(c, Cc, Y[u]) + X[u] * sizeof(MT);
        *reinterpret_cast<MT *>(row + Cc.offD) = MT(0);
        *reinterpret_cast<MT *>(row + Cc.offRho) = rho[u];
        *reinterpret_cast<MT *>(row + Cc.offR) = acc;
      }
    }
  }
}
template <class MT>
__device__ void cRestrict(const CCtx &c, const CLevel<MT> &Fr, const CLevel<MT> &Cr) {
  const CLevel<MT> F = Fr, Cc = Cr;
  if (cIdle(F))
    return;
  if (F.small)
    cRestrictT<true, 1>(c, F, Cc);
  else
    cRestrictT<false, 1>(c, F, Cc);
  cSync(F);
}

// The coarse correction added to the fine nodes of colour 0: those of colour 1,
// with which the sweeps that follow begin, are formed anew from their neighbours.
// (U: fine nodes of a thread side by side)
// kCo: from the rows that cStageCoarse has put in place.
template <bool kS, bool kCo, int U, class MT>
__device__ __forceinline__ void cProlongT(const CCtx &c, const CLevel<MT> &F,
                                          const CLevel<MT> &Cc) {
  int r0, r1;
  cOwnRows(c, F, r0, r1);
  const int half = (F.nx + 1) / 2, cnt = half * (r1 - r0), stride = cStride(F);
  const int Ya = kCo ? cTab<int>(c, F.offPyI)[min(r0, F.ny - 1)] : 0; // the first staged row
  for (int t0 = threadIdx.x; t0 < cnt; t0 += U * stride) {
    int i[U], X0[U], Y0[U];
    bool on[U];
    MT wx[U], wy[U], v[U][4], d[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int t = t0 + u * stride < cnt ? t0 + u * stride : t0;
      const int ly = F.byHalf.div(t), x = 2 * (t - ly * half) + ((r0 + ly) & 1);
      on[u] = t0 + u * stride < cnt && x < F.nx;
      const int xx = x < F.nx ? x : 0;
      i[u] = ly * F.nx + xx;
      X0[u] = cTab<int>(c, F.offPxI)[xx];
      Y0[u] = cTab<int>(c, F.offPyI)[r0 + ly];
      wx[u] = (MT)cTab<float>(c, F.offPxW)[xx];
      wy[u] = (MT)cTab<float>(c, F.offPyW)[r0 + ly];
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int q = *reinterpret_cast<const uint8_t *>(c.smem + F.offCls + i[u]);
      const bool bx = wx[u] < MT(1), by = wy[u] < MT(1);
      auto coarse = [&](int Y) {
        return kCo ? cTab<MT>(c, F.offCo) + (Y - Ya) * Cc.nx
                   : reinterpret_cast<const MT *>(cCoarseRow<kS>(c, Cc, Y) + Cc.offD);
      };
      const MT *c0 = coarse(Y0[u]) + X0[u], *c1 = coarse(Y0[u] + (by ? 1 : 0)) + X0[u];
      v[u][0] = c0[0];
      v[u][1] = bx ? c0[1] : MT(0);
      v[u][2] = by ? c1[0] : MT(0);
      v[u][3] = bx && by ? c1[1] : MT(0);
      d[u] = reinterpret_cast<const MT *>(c.smem + F.offD)[i[u]];
      on[u] = on[u] && reinterpret_cast<const MT *>(c.smem + F.offTab)[8 * q + 6] == MT(0);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      MT s = wx[u] * wy[u] * v[u][0];
      s = fma((MT(1) - wx[u]) * wy[u], v[u][1], s);
      s = fma(wx[u] * (MT(1) - wy[u]), v[u][2], s);
      s = fma((MT(1) - wx[u]) * (MT(1) - wy[u]), v[u][3], s);
      if (on[u])
        reinterpret_cast<MT *>(c.smem + F.offD)[i[u]] = d[u] + s;
    }
  }
}
// The correction of the coarse rows under this CTA's rows, whole rows from wherever
// they live: a prolongation reads each value up to four times, and those of a level
// held by CTA 0 are wanted by every CTA at once.  Measured: 201 x 101 solve 0.2818 ->
// 0.2805 ms, 401 x 201 0.5375 -> 0.5277.
template <class MT>
__device__ __forceinline__ void cStageCoarse(const CCtx &c, const CLevel<MT> &F,
                                             const CLevel<MT> &Cc) {
  int r0, r1;
  cOwnRows(c, F, r0, r1);
  if (r0 >= r1)
    return;
  const int Ya = cTab<int>(c, F.offPyI)[r0];
  const int Yb = min(Cc.ny - 1, cTab<int>(c, F.offPyI)[r1 - 1] + 1);
  MT *co = reinterpret_cast<MT *>(c.smem + F.offCo);
  for (int k = threadIdx.x; k < (Yb - Ya + 1) * Cc.nx; k += kClusterThreads) {
    const int q = Cc.byNx.div(k);
    co[k] = reinterpret_cast<const MT *>(cCoarseRow<false>(c, Cc, Ya + q) + Cc.offD)[k - q * Cc.nx];
  }
}
template <class MT>
__device__ void cProlong(const CCtx &c, const CLevel<MT> &Fr, const CLevel<MT> &Cr) {
  const CLevel<MT> F = Fr, Cc = Cr;
  if (cIdle(F))
    return;
  if (F.small) {
    cProlongT<true, false, 1>(c, F, Cc);
  } else if (F.offCo) {
    cStageCoarse(c, F, Cc);
    __syncthreads();
    cProlongT<false, true, 2>(c, F, Cc);
  } else {
    cProlongT<false, false, 2>(c, F, Cc);
  }
  cSync(F);
}

// coarsest level (held by CTA 0): red-black sweeps, in the registers of warp 0
// when it has at most 32 nodes, else by the threads of the level (warp 0 or the
// block) with their barriers
template <class MT> __device__ void cCoarse(const CCtx &c, const CLevel<MT> &L, int sweeps) {
  if (cIdle(L))
    return;
  const int n = L.nx * L.ny;
  if (n <= 32) {
    if (threadIdx.x < 32) {
      const int i = threadIdx.x, x = i % L.nx, y = i / L.nx;
      const bool live = i < n;
      const Coef<MT> K = cCoef(c, L, live ? cOwn<uint8_t>(c, L, L.offCls, y)[x] : 0);
      MT *dp = live ? cOwn<MT>(c, L, L.offD, y) + x : nullptr;
      const MT r = live ? cOwn<MT>(c, L, L.offR, y)[x] : MT(0);
      const MT den = live ? fma(K.area, cOwn<MT>(c, L, L.offRho, y)[x], K.diag0) : MT(1);
      const MT inv = mgRcp(den);
      const bool upd = live && K.fixed == MT(0);
      MT d = live ? *dp : MT(0);
      // (beyond the domain's edge the coefficient is zero)
      const int lw = (i + 31) & 31, le = (i + 1) & 31, ls = (i - L.nx + 32) & 31,
                ln = (i + L.nx) & 31;
      const bool upd0 = upd && ((x + y) & 1) == 0, upd1 = upd && ((x + y) & 1) == 1;
      for (int it = 0; it < 2 * sweeps; it++) {
        const MT dw = __shfl_sync(0xffffffffu, d, lw), de = __shfl_sync(0xffffffffu, d, le);
        const MT ds = __shfl_sync(0xffffffffu, d, ls), dn = __shfl_sync(0xffffffffu, d, ln);
        const MT s = fma(K.cn, dn, fma(K.cs, ds, fma(K.ce, de, fma(K.cw, dw, r))));
        d = (it & 1 ? upd1 : upd0) ? s * inv : d;
      }
      if (live)
        *dp = d;
    }
    cSync(L);
    return;
  }
  const int stride = cStride(L);
  for (int it = 0; it < sweeps; it++) {
    for (int color = 0; color < 2; color++) {
      for (int i = threadIdx.x; i < n; i += stride) {
        const int x = i % L.nx, y = i / L.nx;
        const Coef<MT> K = cCoef(c, L, cOwn<uint8_t>(c, L, L.offCls, y)[x]);
        if (((x + y) & 1) != color || K.fixed != MT(0))
          continue;
        MT *d = cOwn<MT>(c, L, L.offD, y);
        MT s = cOwn<MT>(c, L, L.offR, y)[x];
        if (x > 0)
          s = fma(K.cw, d[x - 1], s);
        if (x < L.nx - 1)
          s = fma(K.ce, d[x + 1], s);
        if (y > 0)
          s = fma(K.cs, cOwn<MT>(c, L, L.offD, y - 1)[x], s);
        if (y < L.ny - 1)
          s = fma(K.cn, cOwn<MT>(c, L, L.offD, y + 1)[x], s);
        d[x] = s * mgRcp(fma(K.area, cOwn<MT>(c, L, L.offRho, y)[x], K.diag0));
      }
      cSync(L);
    }
  }
}

// max over the block, then over the cluster (every thread of every CTA gets it);
// each CTA's two block maxima sit at byte offset offRed of its shared memory
__device__ __forceinline__ void cClusterMax2(const CCtx &c, unsigned offRed, double &a,
                                             double &b, double *sh) {
  // non-negative values: maxima of their bit patterns (integer instructions;
  // the double-precision pipes are narrow)
  unsigned long long ua = (unsigned long long)__double_as_longlong(a) & ~(1ull << 63);
  unsigned long long ub = (unsigned long long)__double_as_longlong(b) & ~(1ull << 63);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ua = bitsMax(ua, __shfl_xor_sync(0xffffffffu, ua, o));
    ub = bitsMax(ub, __shfl_xor_sync(0xffffffffu, ub, o));
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nW = (int)(blockDim.x >> 5);
  unsigned long long *shu = reinterpret_cast<unsigned long long *>(sh);
  if (lane == 0) {
    shu[2 * w] = ua;
    shu[2 * w + 1] = ub;
  }
  __syncthreads();
  if (w == 0) {
    ua = lane < nW ? shu[2 * lane] : 0ull;
    ub = lane < nW ? shu[2 * lane + 1] : 0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ua = bitsMax(ua, __shfl_xor_sync(0xffffffffu, ua, o));
      ub = bitsMax(ub, __shfl_xor_sync(0xffffffffu, ub, o));
    }
    if (lane == 0) {
      unsigned long long *red = reinterpret_cast<unsigned long long *>(c.smem + offRed);
      red[0] = ua;
      red[1] = ub;
    }
  }
  cg::this_cluster().sync();
  // every warp: lane r reads rank r's maxima, then the warp reduces them
  const int ranks = (int)cg::this_cluster().num_blocks();
  ua = 0ull;
  ub = 0ull;
  for (int r = lane; r < ranks; r += 32) {
    const unsigned long long *o =
        reinterpret_cast<const unsigned long long *>(c.base[r] + offRed);
    ua = bitsMax(ua, o[0]);
    ub = bitsMax(ub, o[1]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ua = bitsMax(ua, __shfl_xor_sync(0xffffffffu, ua, o));
    ub = bitsMax(ub, __shfl_xor_sync(0xffffffffu, ub, o));
  }
  a = __longlong_as_double((long long)ua);
  b = __longlong_as_double((long long)ub);
}

// One V-cycle over the descriptor's levels: the distributed levels, then those
// held by CTA 0, and back up.
template <bool kCol, class MT>
__device__ __forceinline__ void cVcycle(const CCtx &c, const CMG<MT> &M,
                                        cg::cluster_group &cluster) {
  // the distributed levels down ...
  const int Ls = M.firstSmall;
  for (int l = 0; l < Ls; l++) {
    cSmoothSweeps<kCol>(c, M.L[l], M.pre, 0, true);
    cRestrict(c, M.L[l], M.L[l + 1]);
  }
  // ... the levels held by CTA 0 ...
  if (c.rank == 0) {
    for (int l = Ls; l + 1 < M.nLev; l++) {
      cSmoothSweeps<kCol>(c, M.L[l], M.pre, 0, true);
      cRestrict(c, M.L[l], M.L[l + 1]);
    }
    cCoarse(c, M.L[M.nLev - 1], M.coarseSweeps);
    for (int l = M.nLev - 2; l >= Ls; l--) {
      // the CTA reads what warp 0 wrote on the level below
      if (M.L[l + 1].warp && !M.L[l].warp)
        __syncthreads();
      cProlong(c, M.L[l], M.L[l + 1]);
      cSmoothSweeps<kCol>(c, M.L[l], M.post, 1);
    }
  }
  cluster.sync();
  // ... and the distributed levels up
  for (int l = Ls - 1; l >= 0; l--) {
    cProlong(c, M.L[l], M.L[l + 1]);
    cSmoothSweeps<kCol>(c, M.L[l], M.post, 1);
  }
}

// The whole solve: out[0] = final relative residual, out[1] = Newton steps done,
// out[2] = 1 if the update rule stopped the solve.  kTail: one V-cycle of the
// levels below those that the multi-launch path works one launch per phase
// (grids whose finest levels do not fit in shared memory): right-hand side and
// reaction tailR, tailRho of the descriptor's first level, its correction, from
// zero, to tailD.  bad (may be NULL): not zero, the level tables are incomplete
// and nothing is done (out[2] = -1).
template <class MT, bool kTail, bool kCol>
__global__ void __launch_bounds__(kClusterThreads, 1)
    poissonClusterKernel(CMG<MT> Mp, double *__restrict__ pot, const double *__restrict__ conc,
                         const double *__restrict__ C, const double *__restrict__ gSum,
                         const double *__restrict__ gV, double hF0, double hF1, double hP,
                         double rtol, int maxCycles, double updTol,
                         const double *__restrict__ expG, double *__restrict__ out,
                         const MT *__restrict__ tailR, const MT *__restrict__ tailRho,
                         MT *__restrict__ tailD, const int *__restrict__ bad) {
  extern __shared__ __align__(16) char smem[];
  __shared__ char *sBase[kMaxCluster];
  __shared__ double sh[2 * (kClusterThreads / 32)];
  // the level descriptors, read by every phase, from shared memory rather than
  // the parameter bank
  __shared__ __align__(16) int sM[sizeof(CMG<MT>) / sizeof(int)];
  __shared__ __align__(16) double sExp[kExpTab]; // 2^(j/256) for expTab
  if (!kTail && bad && *bad) { // the same for every CTA
    if (blockIdx.x == 0 && threadIdx.x == 0)
      out[2] = -1.;
    return;
  }
  // Staging.  The exp table and level 0's coefficient classes, which the first
  // residual needs, come first; the rest (first needed by the V-cycle) is fetched
  // beside it (stageRest).
  const unsigned sBaseAddr = (unsigned)__cvta_generic_to_shared(smem);
  if (!kTail) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(sExp);
    for (int k = threadIdx.x; k < kExpTab / 2; k += blockDim.x)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a + 16u * k),
                   "l"(expG + 2 * k)
                   : "memory");
  }
  for (int k = threadIdx.x; k < (int)(sizeof(CMG<MT>) / sizeof(int)); k += blockDim.x)
    sM[k] = reinterpret_cast<const int *>(&Mp)[k];
  __syncthreads();
  const CMG<MT> &M = *reinterpret_cast<const CMG<MT> *>(sM);
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
  if (threadIdx.x < ranks)
    sBase[threadIdx.x] = static_cast<char *>(cluster.map_shared_rank((void *)smem, threadIdx.x));
  // n words from src to byte off, by the threads t0, t0 + stride, ...
  auto stage = [&](unsigned off, const void *src, int n, int t0, int stride) {
    const int *sp = static_cast<const int *>(src);
    for (int k = t0; k < n; k += stride)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sBaseAddr + off + 4u * k),
                   "l"(sp + k)
                   : "memory");
  };
  int clsEnd[16]; // prefix sums of this CTA's class bytes per level
  {
    int nCls = 0;
    for (int l = 0; l < M.nLev; l++) {
      const CLevel<MT> &L = M.L[l];
      int r0, r1;
      cOwnRows(CCtx{sBase, smem, rank}, L, r0, r1);
      nCls += L.nx * (r1 - r0);
      clsEnd[l] = nCls;
    }
  }
  stage(M.L[0].offTab, M.L[0].tab, 8 * M.L[0].nCls * (int)(sizeof(MT) / 4), threadIdx.x,
        blockDim.x);
  // this CTA's class bytes of the levels [clsEnd[l0 - 1], clsEnd[l1 - 1]), four
  // bytes per thread and pass: the loads first, then the stores
  auto copyCls = [&](int l0, int l1) {
    const int begin = l0 > 0 ? clsEnd[l0 - 1] : 0, end = clsEnd[l1 - 1];
    for (int t0 = begin + (int)threadIdx.x; t0 < end; t0 += 4 * blockDim.x) {
      uint8_t v[4];
      uint8_t *dst[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int t = t0 + j * (int)blockDim.x;
        dst[j] = nullptr;
        if (t < end) {
          int l = l0;
          while (t >= clsEnd[l])
            l++;
          const CLevel<MT> &L = M.L[l];
          const int k = t - (l > 0 ? clsEnd[l - 1] : 0);
          const int r0 = L.small ? 0 : min(L.ny, rank * L.rowsPer);
          v[j] = L.cls[(size_t)r0 * L.nx + k];
          dst[j] = reinterpret_cast<uint8_t *>(smem + L.offCls) + k;
        }
      }
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (dst[j])
          *dst[j] = v[j];
    }
  };
  copyCls(0, 1);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  // (no cluster barrier yet: the first access to another CTA's shared memory
  // comes after the cluster barrier of the first residual's maxima)
  CCtx c{sBase, smem, rank};
  const CLevel<MT> &L0 = M.L[0];
  const int nx = L0.nx, ny = L0.ny;
  int p0, p1;
  cOwnRows(c, L0, p0, p1);
  const int nOwn = nx * (p1 - p0);
  // the rest of the staging: the class and transfer tables by asynchronous copies, a
  // warp per table (the whole block on each in turn took 6 us to issue), the class
  // bytes of the other levels, zero residuals (Dirichlet nodes keep them); the next
  // cluster barrier makes them visible
  auto stageRest = [&]() {
    for (int a = threadIdx.x >> 5; a < 11 * M.nLev; a += (int)(blockDim.x >> 5)) {
      const int l = a / 11, which = a - 11 * l;
      const CLevel<MT> &L = M.L[l];
      const void *src = L.tab;
      unsigned off = L.offTab;
      int n = l > 0 ? 8 * L.nCls * (int)(sizeof(MT) / 4) : 0;
      if (which > 0 && L.ncx == 0)
        continue;
      switch (which) {
      case 1: src = L.pxIdx, off = L.offPxI, n = L.nx; break;
      case 2: src = L.pxW, off = L.offPxW, n = L.nx; break;
      case 3: src = L.pyIdx, off = L.offPyI, n = L.ny; break;
      case 4: src = L.pyW, off = L.offPyW, n = L.ny; break;
      case 5: src = L.rxIdx, off = L.offRxI, n = 3 * L.ncx; break;
      case 6: src = L.rxW, off = L.offRxW, n = 3 * L.ncx; break;
      case 7: src = L.ryIdx, off = L.offRyI, n = 3 * L.ncy; break;
      case 8: src = L.ryW, off = L.offRyW, n = 3 * L.ncy; break;
      case 9: src = L.mapX, off = L.offMapX, n = L.ncx; break;
      case 10: src = L.mapY, off = L.offMapY, n = L.ncy; break;
      }
      stage(off, src, n, threadIdx.x & 31, 32);
    }
    copyCls(1, M.nLev);
    for (int l = 0; l < M.nLev; l++) { // the padding around d, and rows past the grid's
      const CLevel<MT> &L = M.L[l];
      int r0, r1;
      cOwnRows(c, L, r0, r1);
      const int q = (int)(16 / sizeof(MT));
      MT *d = reinterpret_cast<MT *>(smem + L.offD);
      if ((int)threadIdx.x < q)
        d[(int)threadIdx.x - q] = MT(0);
      for (int k = L.nx * (r1 - r0) + threadIdx.x; k < L.nx * L.rowsPer + q; k += blockDim.x)
        d[k] = MT(0);
    }
    for (int l = 0; l + 1 < M.nLev; l++) {
      const CLevel<MT> &L = M.L[l];
      int r0, r1;
      cOwnRows(c, L, r0, r1);
      MT *res = reinterpret_cast<MT *>(smem + L.offRes);
      for (int k = threadIdx.x; k < L.nx * (r1 - r0); k += blockDim.x)
        res[k] = MT(0);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  };
  if constexpr (kTail) {
    MT *d0 = cOwn<MT>(c, L0, L0.offD, 0);
    MT *r0 = cOwn<MT>(c, L0, L0.offR, 0);
    MT *rho0 = cOwn<MT>(c, L0, L0.offRho, 0);
    for (int t = threadIdx.x; t < nOwn; t += blockDim.x) {
      d0[t] = MT(0);
      r0[t] = tailR[(size_t)p0 * nx + t];
      rho0[t] = tailRho[(size_t)p0 * nx + t];
    }
    stageRest();
    cluster.sync();
    cVcycle<kCol>(c, M, cluster);
    for (int t = threadIdx.x; t < nOwn; t += blockDim.x)
      tailD[(size_t)p0 * nx + t] = d0[t];
    cluster.sync(); // no CTA leaves while another may still read its shared memory
    return;
  }
  double rel = INFINITY, perScale = 1.;
  const bool updRule = updTol > 0.;
  int it = 0;
  bool stopped = false;
  const double c2 = -2.0 * (hF0 + hF1);
  for (;; it++) {
    // F(phi), Jacobian reaction and FV-scaled right-hand side (nonlinResidualKernel);
    // the scale of the relative residual from the first iteration's state
    // Bound by its double-precision instructions on the cluster's few SMs (13 a
    // node): each node's values are loaded while the one before is worked on, and
    // the conversions and comparisons go by bits.  With the staging beside it the
    // 201 x 101 resistor's solve went 0.300 -> 0.283 ms, 401 x 201 0.613 -> 0.568.
    MT aFm = 0;
    double sc = 0.;
    auto load = [&](int t) {
      const int ly = L0.byNx.div(t), y = p0 + ly, x = t - ly * nx;
      return nodeLoad(pot, conc, C, gSum, gV, y * nx + x, x, y, nx, ny);
    };
    // of each scheduler's warps half do their part of the staging first: the
    // double-precision pipe has the other half's nodes meanwhile
    const int residualPart = it == 0 ? (int)(threadIdx.x >> 7) & 1 : 0;
    for (int part = 0; part < 2; part++) {
      if (part != residualPart) {
        if (it == 0)
          stageRest();
        continue;
      }
      NodeIn next;
      if ((int)threadIdx.x < nOwn)
        next = load(threadIdx.x);
      for (int t = threadIdx.x; t < nOwn; t += blockDim.x) {
        const NodeIn in = next;
        next = load(min(t + (int)blockDim.x, nOwn - 1));
        const int ly = L0.byNx.div(t), y = p0 + ly, x = t - ly * nx;
        MT *d0 = cOwn<MT>(c, L0, L0.offD, ly);
        MT *r0 = cOwn<MT>(c, L0, L0.offR, ly);
        MT *rho0 = cOwn<MT>(c, L0, L0.offRho, ly);
        d0[x] = MT(0);
        if (cCoef(c, L0, cOwn<uint8_t>(c, L0, L0.offCls, ly)[x]).fixed != MT(0)) {
          r0[x] = MT(0);
          rho0[x] = MT(0);
          continue;
        }
        const NodeF q = nodeResidual(in, conc != nullptr, hF0, hF1, c2, hP, sExp);
        const double F = q.F, p = q.p, n = q.n;
        const int bd = (x == 0 || x == nx - 1) + (y == 0 || y == ny - 1);
        const MT fF = mgOf<MT>(F);
        r0[x] = fF * (bd == 0 ? MT(1) : (bd == 1 ? MT(0.5) : MT(0.25)));
        rho0[x] = mgOf<MT>(conc ? p : p + n);
        aFm = fmax(aFm, fabs(fF));
        if (it == 0)
          sc = dmaxPos(sc, hP * (fabs(in.C) + n + p));
        // a NaN would vanish in the maxima: non-finite values count as an
        // infinite residual, which ends the solve as not converged
        if (!finiteBits(F) || !finiteBits(p) || !finiteBits(n) || !isfinite(fF))
          aFm = MT(INFINITY);
      }
    }
    double aF = (double)aFm;
    // its cluster barrier also orders the writes above; the maxima are next
    // written after the V-cycle's barriers, when every CTA has read them
    cClusterMax2(c, M.offRed, aF, sc, sh);
    if (it == 0)
      perScale = bitsPositive(sc) ? 1. / sc : 1.;
    // (every warp takes this decision: comparisons by the bit patterns)
    rel = aF * perScale;
    if (!bitsBelow(rtol, rel) || it == maxCycles || !finiteBits(rel))
      break;
    // under the update-size rule a Newton step needs only a rough correction
    const int nv = !updRule && bitsBelow(rel, M.twoCycleRel) ? M.vcycles : 1;
    for (int vc = 0; vc < nv; vc++)
      cVcycle<kCol>(c, M, cluster);
    // clamped Newton update of this CTA's rows (updatePotKernel); the cluster
    // barrier makes the new values visible to the neighbours' next residual
    MT updM = 0;
    constexpr int U = 4; // nodes of a thread side by side
    for (int t0 = threadIdx.x; t0 < nOwn; t0 += U * blockDim.x) {
      double phi[U];
#pragma unroll
      for (int u = 0; u < U; u++)
        phi[u] = pot[(size_t)p0 * nx + min(t0 + u * (int)blockDim.x, nOwn - 1)];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int t = t0 + u * (int)blockDim.x;
        if (t >= nOwn ||
            cCoef(c, L0, cOwn<uint8_t>(c, L0, L0.offCls, 0)[t]).fixed != MT(0))
          continue;
        MT v = cOwn<MT>(c, L0, L0.offD, 0)[t];
        if (isfinite(v)) // a non-finite correction is passed on to the next residual
          v = fmin(MT(kMaxNewtonStep), fmax(MT(-kMaxNewtonStep), v));
        pot[(size_t)p0 * nx + t] = phi[u] + doubleOf(v);
        updM = isfinite(v) ? fmax(updM, fabs(v)) : MT(INFINITY);
      }
    }
    double upd = (double)updM;
    if (updRule) {
      // the maxima of this rule use their own slot (offRed + 16)
      double none = 0.;
      cClusterMax2(c, M.offRed + 16, upd, none, sh);
      if (upd < updTol) {
        it++;
        stopped = true;
        break;
      }
    }
    cluster.sync();
  }
  if (rank == 0 && threadIdx.x == 0) {
    out[0] = rel;
    out[1] = (double)it;
    out[2] = stopped ? 1. : 0.;
  }
  cluster.sync(); // no CTA leaves while another may still read its shared memory
}

// Level layout of the cluster solve for CL CTAs; *bytes = dynamic shared memory,
// 0 if some level has too many coefficient classes.  evenRows: a distributed
// level followed by another gets an even number of rows per CTA, so that a
// CTA's coarse rows lie under its fine rows; without it the bands of two
// levels may be a row apart, and a restriction or prolongation then reaches a
// neighbour's row through distributed shared memory (the same arithmetic, a
// row less per CTA and level: the 401 x 201 grid fits in 12 CTAs).
struct MGSet { // a hierarchy and its cycle
  const MGLevel *L;
  int nLev, pre, post, coarseSweeps, vcycles;
  double twoCycleRel;
};
inline MGSet mgSet(const PoissonMG &P, int first = 0) {
  return {P.L.data() + first, (int)P.L.size() - first, P.pre, P.post, P.coarseSweeps,
          P.vcyclesPerNewton, P.twoCycleRel};
}

// a layout of b bytes beside the kernel's static shared memory: the level
// descriptors, the exp table and the reduction slots
template <class MT> bool clusterSmemFits(size_t b) {
  return b != 0 && b + sizeof(CMG<MT>) + kExpTab * sizeof(double) + 1024 <= kClusterSmemMax;
}

template <class MT>
CMG<MT> clusterDesc(const MGSet &P, int CL, size_t *bytes, bool evenRows = true) {
  CMG<MT> M;
  std::memset(&M, 0, sizeof(M));
  M.nLev = P.nLev;
  M.pre = P.pre;
  M.post = P.post;
  M.coarseSweeps = P.coarseSweeps;
  M.vcycles = P.vcycles;
  M.twoCycleRel = P.twoCycleRel;
  M.firstSmall = M.nLev - 1;
  *bytes = 0;
  for (int l = 0; l < M.nLev; l++) {
    if (P.L[l].nCls <= 0)
      return M;
    const bool small = CL == 1 || P.L[l].nx * P.L[l].ny <= kSmallNodes || l == M.nLev - 1;
    if (small && l < M.firstSmall)
      M.firstSmall = l;
  }
  for (int l = 0; l < M.nLev; l++) {
    CLevel<MT> &c = M.L[l];
    c.nx = P.L[l].nx;
    c.ny = P.L[l].ny;
    c.small = l >= M.firstSmall ? 1 : 0;
    c.warp = l >= 1 && c.small && c.nx * c.ny <= kWarpNodes ? 1 : 0;
  }
  // bands: level 0 split evenly (rounded to even rows when a distributed
  // level follows), each next distributed level on half the rows of the level
  // above where that covers it, else split evenly
  const int B = M.firstSmall - 1;
  for (int l = 0; l <= B; l++) {
    CLevel<MT> &c = M.L[l];
    const int even = (c.ny + CL - 1) / CL;
    int rows = even;
    if (l > 0 && M.L[l - 1].ny > 3 && M.L[l - 1].rowsPer / 2 * CL >= c.ny)
      rows = M.L[l - 1].rowsPer / 2;
    if (evenRows && l < B && (rows & 1))
      rows++;
    c.rowsPer = rows;
  }
  size_t off = 0;
  auto take = [&](size_t b) {
    const size_t o = off;
    off += (b + 15) & ~size_t(15);
    return (unsigned)o;
  };
  // `staged` levels from the finest on have room for the coarse rows under a band
  auto layout = [&](int staged) {
    off = 0;
    for (int l = 0; l < M.nLev; l++) {
      const MGLevel &v = P.L[l];
      CLevel<MT> &c = M.L[l];
      if (c.small)
        c.rowsPer = c.ny;
      c.byNx.set(c.nx);
      c.byHalf.set((c.nx + 1) / 2);
      c.byRows.set(c.rowsPer);
      const size_t cells = (size_t)c.rowsPer * c.nx;
      // zeroed padding before and after d: the sweeps read past the ends of its first
      // and last rows
      take(16);
      c.offD = take(cells * sizeof(MT) + 16);
      c.offR = take(cells * sizeof(MT));
      c.offRho = take(cells * sizeof(MT));
      c.offRes = l + 1 < M.nLev ? take(cells * sizeof(MT)) : 0;
      c.offCls = take(cells);
      c.nCls = v.nCls;
      c.offTab = take((size_t)8 * v.nCls * sizeof(MT));
      // fine rows 2 Y and 2 Y + 1 lie over coarse row Y (rows not coarsened: one each)
      c.offCo = 0;
      if (!c.small && l < staged)
        c.offCo = take((size_t)((P.L[l + 1].ny < c.ny ? c.rowsPer / 2 : c.rowsPer) + 3) *
                       P.L[l + 1].nx * sizeof(MT));
      c.cls = v.cls;
      c.tab = static_cast<const MT *>(v.clsTab);
      if (l + 1 < M.nLev) {
        c.ncx = P.L[l + 1].nx;
        c.ncy = P.L[l + 1].ny;
        c.offPxI = take(4 * (size_t)c.nx);
        c.offPxW = take(4 * (size_t)c.nx);
        c.offPyI = take(4 * (size_t)c.ny);
        c.offPyW = take(4 * (size_t)c.ny);
        c.offRxI = take(12 * (size_t)c.ncx);
        c.offRxW = take(12 * (size_t)c.ncx);
        c.offRyI = take(12 * (size_t)c.ncy);
        c.offRyW = take(12 * (size_t)c.ncy);
        c.offMapX = take(4 * (size_t)c.ncx);
        c.offMapY = take(4 * (size_t)c.ncy);
      }
      c.rxIdx = v.rxIdx;
      c.ryIdx = v.ryIdx;
      c.pxIdx = v.pxIdx;
      c.pyIdx = v.pyIdx;
      c.mapX = v.mapX;
      c.mapY = v.mapY;
      c.rxW = v.rxW;
      c.ryW = v.ryW;
      c.pxW = v.pxW;
      c.pyW = v.pyW;
    }
    M.offRed = take(4 * sizeof(double)); // two slots of two maxima
  };
  layout(M.firstSmall);
  if (!clusterSmemFits<MT>(off))
    layout(0);
  *bytes = off;
  return M;
}

template <class MT> cudaLaunchConfig_t clusterConfig(int CL, size_t bytes, cudaStream_t st,
                                                     cudaLaunchAttribute *at) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CL, 1, 1);
  cfg.blockDim = dim3(kClusterThreads, 1, 1);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = st;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = CL;
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// The kernel of a layout: the one with the column sweeps where a distributed level is
// too large for the others to hold (float); they would slow every other layout's
// kernel by their registers (201 x 101: 0.282 -> 0.289 ms).
template <class MT, bool kTail> auto clusterKernel(const CMG<MT> &M) {
  if constexpr (sizeof(MT) == 4)
    for (int l = 0; l < M.firstSmall; l++)
      if ((M.L[l].nx + 1) / 2 * M.L[l].rowsPer > kSweepNodes * kClusterThreads &&
          columnGroups(M.L[l].nx, M.L[l].rowsPer) > 0)
        return poissonClusterKernel<MT, kTail, sizeof(MT) == 4>;
  return poissonClusterKernel<MT, kTail, false>;
}

// the device's limits taken by a kernel: *maxDyn the dynamic shared memory it may
// have, *bigOk clusters above 8 CTAs.  The memory attribute is one per kernel, shared
// by every hierarchy (engines of other grid sizes), so it is set to the device's
// limit, not to one layout's size.
template <class K> bool clusterOptIn(K k, size_t *maxDyn, bool *bigOk) {
  cudaFuncAttributes fa;
  int dev = 0, optin = 0;
  if (cudaFuncGetAttributes(&fa, k) != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) !=
          cudaSuccess ||
      optin <= (int)fa.sharedSizeBytes ||
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           optin - (int)fa.sharedSizeBytes) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  *maxDyn = std::min(*maxDyn, (size_t)(optin - (int)fa.sharedSizeBytes));
  if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    *bigOk = false;
  }
  return true;
}

// Largest cluster (16, 14, 12, 10, 8, 4, 2 or 1 CTAs, at most P.clusterCap
// when that is set) whose layout fits in shared memory and of which the
// device can hold `concurrent` at once (solves of engines stepped side by
// side); none: the multi-launch path serves the grid.  On GB300 with one
// 512-thread CTA per SM, 16 or 14 CTAs give 7 resident clusters, 12 give 8,
// 10 give 13 and 8 give 15.
struct ClusterFit {
  int size = 0; // CTAs; 0: none fits
  size_t smem = 0;
  bool even = true;
};
template <class MT, bool kTail>
ClusterFit clusterFit(const MGSet &P, int cap, int concurrent) {
  ClusterFit fit;
  const int n = P.L[0].nx * P.L[0].ny;
  size_t maxDyn = kClusterSmemMax;
  bool bigOk = true;
  if (!clusterOptIn(poissonClusterKernel<MT, kTail, false>, &maxDyn, &bigOk))
    return fit;
  if constexpr (sizeof(MT) == 4)
    if (!clusterOptIn(poissonClusterKernel<MT, kTail, true>, &maxDyn, &bigOk))
      return fit;
  const int cands[] = {16, 14, 12, 10, 8, 4, 2, 1};
  for (int CL : cands) {
    if (cap > 0 && CL > cap)
      continue;
    if (CL > 1 && n <= kSmallNodes)
      continue;
    if (CL > 8 && !bigOk)
      continue;
    auto fits = [&](size_t b) { return b <= maxDyn && clusterSmemFits<MT>(b); };
    size_t bytes = 0;
    bool even = true;
    CMG<MT> M = clusterDesc<MT>(P, CL, &bytes, true);
    if (!fits(bytes)) {
      even = false;
      M = clusterDesc<MT>(P, CL, &bytes, false);
      if (!fits(bytes))
        continue;
    }
    cudaLaunchAttribute at;
    cudaLaunchConfig_t cfg = clusterConfig<MT>(CL, bytes, nullptr, &at);
    int nc = 0;
    if (cudaOccupancyMaxActiveClusters(&nc, clusterKernel<MT, kTail>(M), &cfg) != cudaSuccess) {
      cudaGetLastError();
      continue;
    }
    if (nc < std::max(1, concurrent))
      continue;
    fit.size = CL;
    fit.smem = bytes;
    fit.even = even;
    return fit;
  }
  return fit;
}

// The first level whose hierarchy fits in a cluster, below levels that do not
// (0: none, or the whole hierarchy fits): that part of a V-cycle is one launch.
// Measured on 801 x 401 nodes: 135 launches of 4.2 us of host time each per
// V-cycle are 570 us; 15 launches and the cluster of the 401 x 201 hierarchy 140
// us (a solve of 3 Newton steps with its grids in and out 5.50 -> 2.03 ms).
template <class MT> void tailPlan(const MGSet &P, int cap, int &level, ClusterFit &fit) {
  level = 0;
  for (int l = 1; l < P.nLev; l++) {
    MGSet T = P;
    T.L += l;
    T.nLev -= l;
    fit = clusterFit<MT, true>(T, cap, 1);
    if (fit.size) {
      level = l;
      return;
    }
  }
}

template <class MT> void clusterPlan(PoissonMG &P, int concurrent) {
  const ClusterFit f = clusterFit<MT, false>(mgSet(P), P.clusterCap, concurrent);
  P.clusterSize = f.size;
  P.clusterSmem = f.smem;
  P.clusterEven = f.even;
  P.tailLevel = 0;
  if (!f.size && concurrent <= 1) {
    ClusterFit t;
    tailPlan<MT>(mgSet(P), P.clusterCap, P.tailLevel, t);
    P.tailSize = t.size;
    P.tailEven = t.even;
  }
}

} // namespace

int32_t poissonPlanCluster(PoissonMG &P, int concurrent) {
  if (P.L.empty())
    return EMCG_OK;
  if (P.fp32)
    clusterPlan<float>(P, concurrent);
  else
    clusterPlan<double>(P, concurrent);
  // a cap or a concurrency that nothing meets: plan for one solve at a time
  if (P.clusterSize == 0 && concurrent > 1) {
    if (P.fp32)
      clusterPlan<float>(P, 1);
    else
      clusterPlan<double>(P, 1);
  }
  return cudaGetLastError() == cudaSuccess ? EMCG_OK : EMCG_ERR_CUDA;
}

namespace {

// The V-cycle of the levels from P.L on, one launch per phase; tailLevel > 0:
// from that level on in one cluster launch of tailSize CTAs.
struct MGTail {
  int level = 0, size = 0;
  bool even = true;
};
// The tail's launch (its status is the solve's next cudaGetLastError).  A call: its
// descriptors, 8 KB, are not on the stack of every level of the recursion.
template <class MT>
__attribute__((noinline)) void launchTail(const MGSet &P, const LevelK<MT> &K, const MGTail &tail,
                                          cudaStream_t st) {
  MGSet T = P;
  T.L += tail.level;
  T.nLev -= tail.level;
  size_t bytes = 0;
  const CMG<MT> M = clusterDesc<MT>(T, tail.size, &bytes, tail.even);
  cudaLaunchAttribute at;
  cudaLaunchConfig_t cfg = clusterConfig<MT>(tail.size, bytes, st, &at);
  cudaLaunchKernelEx(&cfg, clusterKernel<MT, true>(M), M, (double *)nullptr,
                     (const double *)nullptr, (const double *)nullptr, (const double *)nullptr,
                     (const double *)nullptr, 0., 0., 0., 0., 0, 0., (const double *)nullptr,
                     (double *)nullptr, (const MT *)K.r, (const MT *)K.rho, K.d,
                     (const int *)nullptr);
}
template <class MT>
void vcycle(const MGSet &P, int l, const MGTail &tail, cudaStream_t st) {
  const MGLevel &lv = P.L[l];
  LevelK<MT> K = levelK<MT>(lv);
  const int n = lv.nx * lv.ny;
  if (tail.level && l == tail.level)
    return launchTail<MT>(P, K, tail, st);
  if (l + 1 == P.nLev) {
    coarseSolveKernel<MT><<<1, 256, 0, st>>>(K, P.coarseSweeps);
    return;
  }
  const int half = ((lv.nx + 1) / 2) * lv.ny;
  const int gs = (half + kBlock - 1) / kBlock;
  for (int s = 0; s < P.pre; s++) {
    smoothKernel<MT><<<gs, kBlock, 0, st>>>(K, 0);
    smoothKernel<MT><<<gs, kBlock, 0, st>>>(K, 1);
  }
  const MGLevel &cl = P.L[l + 1];
  LevelK<MT> Kc = levelK<MT>(cl);
  const int nc = cl.nx * cl.ny;
  restrictKernel<MT><<<(nc + kBlock - 1) / kBlock, kBlock, 0, st>>>(
      K, Kc, lv.rxIdx, lv.rxW, lv.ryIdx, lv.ryW, lv.mapX, lv.mapY);
  vcycle<MT>(P, l + 1, tail, st);
  prolongKernel<MT><<<(n + kBlock - 1) / kBlock, kBlock, 0, st>>>(K, Kc, lv.pxIdx, lv.pxW,
                                                                  lv.pyIdx, lv.pyW);
  for (int s = 0; s < P.post; s++) {
    smoothKernel<MT><<<gs, kBlock, 0, st>>>(K, 1);
    smoothKernel<MT><<<gs, kBlock, 0, st>>>(K, 0);
  }
}

// 1-D coarsening: coarse node I sits on fine node min(2I, n-1)
void coarsen1d(int n, std::vector<int> &map) {
  map.clear();
  if (n <= 3) {
    for (int i = 0; i < n; i++)
      map.push_back(i);
    return;
  }
  int nc = (n - 1 + 1) / 2 + 1;
  for (int I = 0; I < nc; I++)
    map.push_back(std::min(2 * I, n - 1));
}

// transfer weights between fine coordinates xf and coarse xc (= xf[map])
void transfer1d(const std::vector<double> &xf, const std::vector<int> &map,
                std::vector<int> &pIdx, std::vector<float> &pW, std::vector<int> &rIdx,
                std::vector<float> &rW) {
  const int nf = (int)xf.size(), nc = (int)map.size();
  pIdx.assign(nf, 0);
  pW.assign(nf, 1.f);
  int I = 0;
  for (int i = 0; i < nf; i++) {
    while (I + 1 < nc && map[I + 1] <= i)
      I++;
    pIdx[i] = I;
    if (map[I] == i || I + 1 >= nc)
      pW[i] = 1.f;
    else
      pW[i] = (float)((xf[map[I + 1]] - xf[i]) / (xf[map[I + 1]] - xf[map[I]]));
  }
  rIdx.assign(3 * nc, 0);
  rW.assign(3 * nc, 0.f);
  std::vector<int> cnt(nc, 0);
  for (int i = 0; i < nf; i++) {
    int J = pIdx[i];
    float w = pW[i];
    if (w > 0.f && cnt[J] < 3) {
      rIdx[3 * J + cnt[J]] = i;
      rW[3 * J + cnt[J]] = w;
      cnt[J]++;
    }
    if (w < 1.f && J + 1 < nc && cnt[J + 1] < 3) {
      rIdx[3 * (J + 1) + cnt[J + 1]] = i;
      rW[3 * (J + 1) + cnt[J + 1]] = 1.f - w;
      cnt[J + 1]++;
    }
  }
}

template <class V> int32_t upload(V **dst, const std::vector<V> &src, cudaStream_t st) {
  EMCG_CUDA(cudaMalloc(dst, sizeof(V) * std::max<size_t>(src.size(), 1)));
  if (!src.empty())
    EMCG_CUDA(cudaMemcpyAsync(*dst, src.data(), sizeof(V) * src.size(), cudaMemcpyHostToDevice, st));
  return EMCG_OK;
}

// Distinct coefficient tuples of a level (a uniform grid has a handful:
// interior, edges, corners, contacts, gates) and each node's class.
template <class MT>
int32_t coefficientClasses(MGLevel &L, const std::vector<double> &cw,
                           const std::vector<double> &ce, const std::vector<double> &cs,
                           const std::vector<double> &cn, const std::vector<double> &ar,
                           const std::vector<double> &dg, const std::vector<uint8_t> &fixed,
                           cudaStream_t st) {
  const size_t m = cw.size();
  std::vector<uint8_t> cls(m);
  std::vector<MT> tab;
  std::map<std::array<MT, 7>, int> ids;
  for (size_t k = 0; k < m && L.nCls >= 0; k++) {
    std::array<MT, 7> t = {(MT)cw[k], (MT)ce[k], (MT)cs[k], (MT)cn[k],
                           (MT)ar[k], (MT)dg[k], (MT)(fixed[k] ? 1 : 0)};
    auto it = ids.find(t);
    if (it == ids.end()) {
      if (ids.size() == 255) {
        L.nCls = -1;
        break;
      }
      it = ids.emplace(t, (int)ids.size()).first;
      tab.insert(tab.end(), t.begin(), t.end());
      tab.push_back(MT(0));
    }
    cls[k] = (uint8_t)it->second;
  }
  if (L.nCls < 0) {
    L.nCls = 0;
    return EMCG_OK;
  }
  L.nCls = (int)ids.size();
  EMCG_TRY(upload(&L.cls, cls, st));
  MT *t = nullptr;
  EMCG_TRY(upload(&t, tab, st));
  L.clsTab = t;
  return EMCG_OK;
}

} // namespace

int32_t poissonCreate(PoissonMG &P, const PoissonSetup &S, bool fp32, int smooth,
                      cudaStream_t st) {
  P.S = S;
  P.fp32 = fp32;
  if (smooth > 0)
    P.pre = P.post = smooth;
  const int nx = S.nx, ny = S.ny;
  P.hF[0] = S.h[1] / S.h[0];
  P.hF[1] = S.h[0] / S.h[1];
  P.hP = 1.;
  P.hP = P.hP * S.h[0];
  P.hP = P.hP * S.h[1];
  EMCG_TRY(upload(&P.C, S.C, st));
  EMCG_TRY(upload(&P.gSum, S.gSum, st));
  EMCG_TRY(upload(&P.gVeq, S.gVeq, st));
  EMCG_TRY(upload(&P.gVne, S.gVne, st));
  EMCG_TRY(upload(&P.resetMask, S.resetMask, st));
  EMCG_TRY(upload(&P.resetEq, S.resetEq, st));
  EMCG_TRY(upload(&P.resetNe, S.resetNe, st));
  EMCG_CUDA(cudaMalloc(&P.stats, 3 * sizeof(double)));
  EMCG_CUDA(cudaMalloc(&P.expTab, kExpTab * sizeof(double)));
  expTableKernel<<<1, kExpTab, 0, st>>>(P.expTab);
  EMCG_CUDA(cudaGetLastError());
  // level hierarchy (host)
  std::vector<double> X(nx), Y(ny);
  for (int i = 0; i < nx; i++)
    X[i] = i * S.h[0];
  for (int j = 0; j < ny; j++)
    Y[j] = j * S.h[1];
  std::vector<uint8_t> fixed = S.fixed;
  std::vector<double> gx = S.gDensX, gy = S.gDensY;
  int lx = nx, ly = ny;
  for (int lev = 0; lev < 16; lev++) {
    MGLevel L;
    std::memset(&L, 0, sizeof(L));
    L.nx = lx;
    L.ny = ly;
    const int m = lx * ly;
    std::vector<double> cw(m), ce(m), cs(m), cn(m), ar(m), dg(m);
    for (int j = 0; j < ly; j++)
      for (int i = 0; i < lx; i++) {
        int k = j * lx + i;
        double dxw = i > 0 ? X[i] - X[i - 1] : 0, dxe = i < lx - 1 ? X[i + 1] - X[i] : 0;
        double dys = j > 0 ? Y[j] - Y[j - 1] : 0, dyn = j < ly - 1 ? Y[j + 1] - Y[j] : 0;
        double lxd = 0.5 * (dxw + dxe), lyd = 0.5 * (dys + dyn);
        cw[k] = i > 0 ? lyd / dxw : 0;
        ce[k] = i < lx - 1 ? lyd / dxe : 0;
        cs[k] = j > 0 ? lxd / dys : 0;
        cn[k] = j < ly - 1 ? lxd / dyn : 0;
        ar[k] = lxd * lyd;
        dg[k] = cw[k] + ce[k] + cs[k] + cn[k] + gx[k] * lyd + gy[k] * lxd;
      }
    if (fp32) {
      auto f = [](const std::vector<double> &v) { return std::vector<float>(v.begin(), v.end()); };
      EMCG_TRY(upload(&L.cw, f(cw), st));
      EMCG_TRY(upload(&L.ce, f(ce), st));
      EMCG_TRY(upload(&L.cs, f(cs), st));
      EMCG_TRY(upload(&L.cn, f(cn), st));
      EMCG_TRY(upload(&L.area, f(ar), st));
      EMCG_TRY(upload(&L.diag0, f(dg), st));
      EMCG_CUDA(cudaMalloc(&L.d, sizeof(float) * m));
      EMCG_CUDA(cudaMalloc(&L.r, sizeof(float) * m));
      EMCG_CUDA(cudaMalloc(&L.rho, sizeof(float) * m));
    } else {
      EMCG_TRY(upload(&L.dcw, cw, st));
      EMCG_TRY(upload(&L.dce, ce, st));
      EMCG_TRY(upload(&L.dcs, cs, st));
      EMCG_TRY(upload(&L.dcn, cn, st));
      EMCG_TRY(upload(&L.darea, ar, st));
      EMCG_TRY(upload(&L.ddiag0, dg, st));
      EMCG_CUDA(cudaMalloc(&L.dd, sizeof(double) * m));
      EMCG_CUDA(cudaMalloc(&L.dr, sizeof(double) * m));
      EMCG_CUDA(cudaMalloc(&L.drho, sizeof(double) * m));
    }
    EMCG_TRY(upload(&L.fixed, fixed, st));
    EMCG_TRY(fp32 ? coefficientClasses<float>(L, cw, ce, cs, cn, ar, dg, fixed, st)
                  : coefficientClasses<double>(L, cw, ce, cs, cn, ar, dg, fixed, st));
    std::vector<int> mx, my;
    coarsen1d(lx, mx);
    coarsen1d(ly, my);
    bool last = (int)mx.size() == lx && (int)my.size() == ly;
    if (!last) {
      std::vector<int> pxI, pyI, rxI, ryI;
      std::vector<float> pxW, pyW, rxW, ryW;
      transfer1d(X, mx, pxI, pxW, rxI, rxW);
      transfer1d(Y, my, pyI, pyW, ryI, ryW);
      EMCG_TRY(upload(&L.pxIdx, pxI, st));
      EMCG_TRY(upload(&L.pyIdx, pyI, st));
      EMCG_TRY(upload(&L.pxW, pxW, st));
      EMCG_TRY(upload(&L.pyW, pyW, st));
      EMCG_TRY(upload(&L.rxIdx, rxI, st));
      EMCG_TRY(upload(&L.ryIdx, ryI, st));
      EMCG_TRY(upload(&L.rxW, rxW, st));
      EMCG_TRY(upload(&L.ryW, ryW, st));
      EMCG_TRY(upload(&L.mapX, mx, st));
      EMCG_TRY(upload(&L.mapY, my, st));
    }
    P.L.push_back(L);
    if (last)
      break;
    // next level's static data by injection
    std::vector<double> Xc(mx.size()), Yc(my.size());
    for (size_t I = 0; I < mx.size(); I++)
      Xc[I] = X[mx[I]];
    for (size_t J = 0; J < my.size(); J++)
      Yc[J] = Y[my[J]];
    const int ncx = (int)mx.size(), ncy = (int)my.size();
    std::vector<uint8_t> fc(ncx * ncy);
    std::vector<double> gxc(ncx * ncy), gyc(ncx * ncy);
    for (int J = 0; J < ncy; J++)
      for (int I = 0; I < ncx; I++) {
        int k = my[J] * lx + mx[I];
        fc[J * ncx + I] = fixed[k];
        gxc[J * ncx + I] = gx[k];
        gyc[J * ncx + I] = gy[k];
      }
    X = Xc;
    Y = Yc;
    fixed = fc;
    gx = gxc;
    gy = gyc;
    lx = ncx;
    ly = ncy;
  }
  EMCG_CUDA(cudaStreamSynchronize(st));
  return poissonPlanCluster(P, 1);
}

void poissonFree(PoissonMG &P) {
  for (auto &L : P.L) {
    void *ps[] = {L.cw,  L.ce,    L.cs,    L.cn,    L.area,  L.diag0, L.dcw,   L.dce,
                  L.dcs, L.dcn,   L.darea, L.ddiag0, L.fixed, L.d,     L.r,     L.rho,
                  L.dd,  L.dr,    L.drho,  L.rxIdx, L.ryIdx, L.rxW,   L.ryW,   L.pxIdx,
                  L.pyIdx, L.pxW, L.pyW,   L.mapX,  L.mapY, L.cls, L.clsTab};
    for (void *p : ps)
      cudaFree(p);
  }
  P.L.clear();
  void *ps[] = {P.C,       P.gSum,    P.gVeq,  P.gVne,  P.resetMask,
                P.resetEq, P.resetNe, P.stats, P.expTab};
  for (void *p : ps)
    cudaFree(p);
  if (P.hStats)
    cudaFreeHost(P.hStats);
  P.hStats = nullptr;
}

// the single-launch cluster solve, enqueued on st
// out: where the kernel writes [relative residual, Newton steps, stopped by
// the update rule] (device memory, or mapped page-locked host memory)
template <class MT>
static int32_t clusterLaunch(PoissonMG &P, double *pot, const double *conc, double rtol,
                             int maxCycles, cudaStream_t st, double *out) {
  size_t bytes = 0;
  const CMG<MT> M = clusterDesc<MT>(mgSet(P), P.clusterSize, &bytes, P.clusterEven);
  cudaLaunchAttribute at;
  cudaLaunchConfig_t cfg = clusterConfig<MT>(P.clusterSize, bytes, st, &at);
  EMCG_CUDA(cudaLaunchKernelEx(&cfg, clusterKernel<MT, false>(M), M, pot, conc,
                               (const double *)P.C, (const double *)P.gSum,
                               (const double *)(conc ? P.gVne : P.gVeq), P.hF[0], P.hF[1], P.hP,
                               rtol, maxCycles, P.updTol, (const double *)P.expTab, out,
                               (const MT *)nullptr, (const MT *)nullptr, (MT *)nullptr,
                               (const int *)nullptr));
  return EMCG_OK;
}

// the outcome of a solve from its statistics
static int32_t solveOutcome(double rel, int it, bool updStop, double rtol, double *relRes,
                            int *cycles) {
  if (relRes)
    *relRes = rel;
  if (cycles)
    *cycles = it;
  if (!std::isfinite(rel)) {
    setError("Poisson: non-finite residual after %d Newton steps (NaN or Inf in the potential, "
             "the concentration or a correction)", it);
    return EMCG_ERR_NONCONVERGED;
  }
  if (!updStop && !(rel <= rtol)) {
    setError("Poisson: relative residual %.3e after %d Newton steps (target %.1e)", rel, it, rtol);
    return EMCG_ERR_NONCONVERGED;
  }
  return EMCG_OK;
}

template <class MT>
static int32_t solveT(PoissonMG &P, double *pot, const double *conc, bool resetBC, double rtol,
                      int maxCycles, cudaStream_t st, double *relRes, int *cycles) {
  const int nx = P.S.nx, ny = P.S.ny, n = nx * ny;
  const int grid = (n + kBlock - 1) / kBlock;
  if (resetBC) {
    resetBCKernel<<<grid, kBlock, 0, st>>>(pot, P.resetMask, conc ? P.resetNe : P.resetEq, n);
    EMCG_CUDA(cudaGetLastError());
  }
  MGLevel &L0 = P.L[0];
  LevelK<MT> K0 = levelK<MT>(L0);
  double stats[3] = {0, 0, 0};
  double rel = INFINITY;
  int it = 0;
  bool updStop = false;
  const bool cluster = P.useCluster && P.clusterSize > 0;
  MGTail tail;
  if (P.useCluster && !cluster && P.tailLevel)
    tail = {P.tailLevel, P.tailSize, P.tailEven};
  if (cluster) {
    EMCG_TRY(clusterLaunch<MT>(P, pot, conc, rtol, maxCycles, st, P.stats));
    EMCG_CUDA(cudaMemcpyAsync(stats, P.stats, 3 * sizeof(double), cudaMemcpyDeviceToHost, st));
    EMCG_CUDA(cudaStreamSynchronize(st));
    rel = stats[0];
    it = (int)stats[1];
    updStop = stats[2] != 0.;
  }
  double scale = 0.;
  for (; !cluster && it <= maxCycles; it++) {
    EMCG_CUDA(cudaMemsetAsync(P.stats, 0, 3 * sizeof(double), st));
    nonlinResidualKernel<MT><<<grid, kBlock, 0, st>>>(
        pot, conc, P.C, L0.fixed, P.gSum, conc ? P.gVne : P.gVeq, nx, ny, P.hF[0], P.hF[1], P.hP,
        K0.r, K0.rho, K0.d, P.stats, it == 0);
    EMCG_CUDA(cudaGetLastError());
    EMCG_CUDA(cudaMemcpyAsync(stats, P.stats, 2 * sizeof(double), cudaMemcpyDeviceToHost, st));
    EMCG_CUDA(cudaStreamSynchronize(st));
    if (it == 0)
      scale = stats[1];
    rel = scale > 0 ? stats[0] / scale : stats[0];
    if (rel <= rtol || it == maxCycles || !std::isfinite(rel))
      break;
    // under the update-size rule a Newton step needs only a rough correction
    const int nv = P.updTol <= 0. && rel < P.twoCycleRel ? P.vcyclesPerNewton : 1;
    for (int k = 0; k < nv; k++)
      vcycle<MT>(mgSet(P), 0, tail, st);
    EMCG_CUDA(cudaGetLastError());
    updatePotKernel<MT><<<grid, kBlock, 0, st>>>(pot, K0.d, L0.fixed, n, P.stats);
    EMCG_CUDA(cudaGetLastError());
    if (P.updTol > 0.) {
      EMCG_CUDA(cudaMemcpyAsync(&stats[2], P.stats + 2, sizeof(double), cudaMemcpyDeviceToHost,
                                st));
      EMCG_CUDA(cudaStreamSynchronize(st));
      if (stats[2] < P.updTol) {
        it++;
        updStop = true;
        break;
      }
    }
  }
  return solveOutcome(rel, it, updStop, rtol, relRes, cycles);
}

int32_t poissonSolve(PoissonMG &P, double *pot, const double *conc, bool resetBC, double rtol,
                     int maxCycles, cudaStream_t st, double *relRes, int *cycles) {
  return P.fp32 ? solveT<float>(P, pot, conc, resetBC, rtol, maxCycles, st, relRes, cycles)
                : solveT<double>(P, pot, conc, resetBC, rtol, maxCycles, st, relRes, cycles);
}

int32_t poissonEnqueue(PoissonMG &P, double *pot, const double *conc, bool resetBC, double rtol,
                       int maxCycles, cudaStream_t st, bool *queued, double *relRes,
                       int *cycles) {
  *queued = false;
  if (!(P.useCluster && P.clusterSize > 0))
    return poissonSolve(P, pot, conc, resetBC, rtol, maxCycles, st, relRes, cycles);
  if (!P.hStats) {
    EMCG_CUDA(cudaHostAlloc(&P.hStats, 3 * sizeof(double), cudaHostAllocMapped));
    EMCG_CUDA(cudaHostGetDevicePointer(&P.hStatsDev, P.hStats, 0));
  }
  if (resetBC) {
    const int n = P.S.nx * P.S.ny;
    resetBCKernel<<<(n + kBlock - 1) / kBlock, kBlock, 0, st>>>(
        pot, P.resetMask, conc ? P.resetNe : P.resetEq, n);
    EMCG_CUDA(cudaGetLastError());
  }
  // the kernel writes its statistics straight into the page-locked block: no
  // copy follows it on the stream
  EMCG_TRY(P.fp32 ? clusterLaunch<float>(P, pot, conc, rtol, maxCycles, st, P.hStatsDev)
                  : clusterLaunch<double>(P, pot, conc, rtol, maxCycles, st, P.hStatsDev));
  *queued = true;
  return EMCG_OK;
}

int32_t poissonFinish(PoissonMG &P, double rtol, double *relRes, int *cycles) {
  EMCG_CHECK_ARG(P.hStats, "no enqueued Poisson solve");
  return solveOutcome(P.hStats[0], (int)P.hStats[1], P.hStats[2] != 0., rtol, relRes, cycles);
}

} // namespace emcg

// ===========================================================================
// Poisson solve that allocates nothing (emcg_poisson_solve_noalloc).
//
// Some callers cannot allocate device memory at the moment they solve: a host
// whose memory pool owns the whole GPU, a caller inside a region where the CUDA
// allocator must not be entered, or an embedder that must not grow the
// process's device footprint after start-up.  For them the solver's working set
// -- fine-grid inputs, the multigrid hierarchy, transfer tables and residual
// statistics -- lives in one file-scope device array of fixed size, reserved
// when this library's device code is loaded.  It is rebuilt from the caller's
// description by kernels on every call; the host side uses only stack memory, of which
// a frame of 31 KB and below it the tail's 8 KB or the levels' recursion.
// Host code cannot pass the array's name to a kernel as an address: the first
// call on each device asks the runtime for the address (cudaGetSymbolAddress,
// with that device current) and keeps it.  The array is shared by all calls,
// so calls whose work can overlap on a device race with one another.
// ===========================================================================
namespace emcg {
namespace {

constexpr int kNAMaxNodes = 1 << 17;           // fine-grid nodes, e.g. 401 x 201 or 362 x 362
constexpr int kNAMaxDim = 8192;                // nodes per dimension
constexpr int kNAMaxLevels = 16;               // as the allocating hierarchy
constexpr int kNAMaxContacts = 64;
// the boundaries' contacts and the contacts' types: a byte each, so that the copy of
// them that the call keeps on its stack is 16 KB (131 KB as int); the longest
// boundary is that of kNAMaxDim nodes by what kNAMaxNodes leaves
constexpr int kNAMaxEdge = 2 * (kNAMaxDim + kNAMaxNodes / kNAMaxDim) + kNAMaxContacts;
static_assert(kNAMaxContacts <= 127, "contacts in a byte");
constexpr int kNAMaxDevices = 64;
constexpr int kNAVcyclesPerNewton = 3; // as PoissonMG's defaults
constexpr double kNATwoCycleRel = 1e30;
constexpr int kNALevelNodes = 2 * kNAMaxNodes; // nodes of all levels together
// coefficient classes per level (a uniform grid has about a dozen, each gate
// a few more); with more the solve runs one launch per phase
constexpr int kNAClasses = 64;
constexpr int kNA1D = 16 * kNAMaxDim;          // 1-D transfer entries of all levels

// byte offsets inside the scratch array
constexpr size_t kOffDoping = 0;                       // double [N]  doping (upload)
constexpr size_t kOffC = kOffDoping + 8ull * kNAMaxNodes;   // double [N]  C = doping / ni
constexpr size_t kOffGSum = kOffC + 8ull * kNAMaxNodes;     // double [N]  gate sums
constexpr size_t kOffGVeq = kOffGSum + 8ull * kNAMaxNodes;
constexpr size_t kOffGVne = kOffGVeq + 8ull * kNAMaxNodes;
constexpr size_t kOffGDx = kOffGVne + 8ull * kNAMaxNodes;   // double [N]  Robin densities
constexpr size_t kOffGDy = kOffGDx + 8ull * kNAMaxNodes;
constexpr size_t kOffResEq = kOffGDy + 8ull * kNAMaxNodes;  // double [N]  resetBC values
constexpr size_t kOffResNe = kOffResEq + 8ull * kNAMaxNodes;
constexpr size_t kOffStats = kOffResNe + 8ull * kNAMaxNodes; // double [4] residual maxima
constexpr size_t kOffLevelF = kOffStats + 256;               // float [9 x all levels]
constexpr size_t kOffTransF = kOffLevelF + 4ull * 9 * kNALevelNodes; // float [1-D]
constexpr size_t kOffTransI = kOffTransF + 4ull * kNA1D;             // int   [1-D]
constexpr size_t kOffBnd = kOffTransI + 4ull * kNA1D;                // i8 [2 (ny + nx) + contacts]
constexpr size_t kOffResMask = kOffBnd + kNAMaxEdge;                 // u8    [N]
constexpr size_t kOffFixed = kOffResMask + kNAMaxNodes;              // u8    [all levels]
constexpr size_t kOffCls = (kOffFixed + kNALevelNodes + 255) & ~size_t(255); // u8 [all levels]
constexpr size_t kOffTab = kOffCls + kNALevelNodes; // float [levels x classes x 8]
constexpr size_t kOffSlot = kOffTab + 32ull * kNAMaxLevels * kNAClasses; // int [levels x classes]
constexpr size_t kOffBad = kOffSlot + 4ull * kNAMaxLevels * kNAClasses;  // int: a table overflowed
constexpr size_t kOffExp = kOffBad + 256;                                // double [exp table]
constexpr size_t kNABytes = (kOffExp + 8ull * kExpTab + 255) & ~size_t(255); // about 21 MB

struct NALevels {
  int n;
  int nx[kNAMaxLevels], ny[kNAMaxLevels];
  double h0, h1; // normalised fine spacing
};

struct NAContacts {
  double gF[kNAMaxContacts], barrier[kNAMaxContacts], volt[kNAMaxContacts];
};

// fine index of node I of level l along one dimension (coarse node I sits on
// node min(2I, n - 1) of the level below while that level has more than 3)
__device__ __forceinline__ int naFineIndex(const NALevels &lv, int l, int I, bool ydim) {
  for (int k = l; k > 0; k--) {
    int nf = ydim ? lv.ny[k - 1] : lv.nx[k - 1];
    if (nf > 3)
      I = min(2 * I, nf - 1);
  }
  return I;
}
__device__ __forceinline__ double naCoord(const NALevels &lv, int l, int I, bool ydim) {
  return naFineIndex(lv, l, I, ydim) * (ydim ? lv.h1 : lv.h0);
}

// Fine-grid data of the reference equation
// (include/PoissonSolver/emcSORSolver.hpp:25-36, 330-368): the same values
// emcg_device_create prepares on the host for the allocating solver.
__global__ void naFineSetupKernel(int nx, int ny, double Ni, double hF0, double hF1, double h0,
                                  double h1, NAContacts ct, const double *doping,
                                  const int8_t *bnd, const int8_t *ctype, double *C,
                                  double *gSum, double *gVeq, double *gVne, double *gDx,
                                  double *gDy, uint8_t *resMask, double *resEq, double *resNe,
                                  uint8_t *fixed) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nx * ny)
    return;
  const int x = i % nx, y = i / nx;
  // boundary b's contact at a node: XMIN/XMAX indexed by y, YMIN/YMAX by x
  auto contact = [&](int b) { return b == 0 ? bnd[y] : b == 1 ? bnd[ny + y]
                                     : b == 2 ? bnd[2 * ny + x] : bnd[2 * ny + nx + x]; };
  const double c = doping[i] / Ni;
  C[i] = c;
  // reservoir nodes: the first boundary holding the node decides
  // (emcSurface::getBoundaryPos, include/emcSurface.hpp)
  int fb = x == 0 ? 0 : (x == nx - 1 ? 1 : (y == 0 ? 2 : (y == ny - 1 ? 3 : -1)));
  int fc = fb < 0 ? -1 : contact(fb);
  fixed[i] = fc >= 0 && ctype[fc] == EMCG_CONTACT_OHMIC;
  // gate Robin terms of every side the node lies on
  const double hF[2] = {hF0, hF1}, h[2] = {h0, h1};
  double gs = 0, ge = 0, gn = 0, dx = 0, dy = 0;
  for (int k = 0; k < 2; k++) {
    int co = k == 0 ? x : y, mx = k == 0 ? nx - 1 : ny - 1;
    for (int side = 0; side < 2; side++) {
      if (co != (side == 0 ? 0 : mx))
        continue;
      int cc = contact(2 * k + side);
      if (cc < 0 || ctype[cc] != EMCG_CONTACT_GATE)
        continue;
      double G = __dmul_rn(__dmul_rn(ct.gF[cc], hF[k]), h[k]);
      gs = __dadd_rn(gs, G);
      ge = __dadd_rn(ge, __dmul_rn(G, ct.barrier[cc]));
      gn = __dadd_rn(gn, __dmul_rn(G, __dadd_rn(ct.barrier[cc], ct.volt[cc])));
      if (k == 0)
        dx = __dadd_rn(dx, 0.5 * ct.gF[cc]);
      else
        dy = __dadd_rn(dy, 0.5 * ct.gF[cc]);
    }
  }
  gSum[i] = gs;
  gVeq[i] = ge;
  gVne[i] = gn;
  gDx[i] = dx;
  gDy[i] = dy;
  // resetBC: every boundary coordinate of an ohmic contact, later boundaries
  // (XMIN, XMAX, YMIN, YMAX order) overriding earlier ones at corners
  uint8_t m = 0;
  double re = 0, rn = 0;
  for (int b = 0; b < 4; b++) {
    bool on = b == 0 ? x == 0 : b == 1 ? x == nx - 1 : b == 2 ? y == 0 : y == ny - 1;
    int cc = on ? contact(b) : -1;
    if (cc < 0 || ctype[cc] != EMCG_CONTACT_OHMIC)
      continue;
    double bi = asinh(0.5 * c);
    m = 1;
    re = bi;
    rn = __dadd_rn(ct.volt[cc], bi);
  }
  resMask[i] = m;
  resEq[i] = re;
  resNe[i] = rn;
}

struct NASet { // the levels' arrays
  MGLevel L[kNAMaxLevels];
};

// finite-volume coefficients and Dirichlet mask of level blockIdx.y, by injection
// of the fine data (the construction poissonCreate runs on the host)
__global__ void naLevelSetupKernel(const __grid_constant__ NALevels lv,
                                   const __grid_constant__ NASet set, const double *gDx,
                                   const double *gDy, const uint8_t *fixed0, int nx0) {
  const int l = blockIdx.y;
  const MGLevel &M = set.L[l];
  const int lx = lv.nx[l], ly = lv.ny[l];
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= lx * ly)
    return;
  const int i = k % lx, j = k / lx;
  const double Xi = naCoord(lv, l, i, false), Yj = naCoord(lv, l, j, true);
  const double dxw = i > 0 ? Xi - naCoord(lv, l, i - 1, false) : 0;
  const double dxe = i < lx - 1 ? naCoord(lv, l, i + 1, false) - Xi : 0;
  const double dys = j > 0 ? Yj - naCoord(lv, l, j - 1, true) : 0;
  const double dyn = j < ly - 1 ? naCoord(lv, l, j + 1, true) - Yj : 0;
  const double lxd = 0.5 * (dxw + dxe), lyd = 0.5 * (dys + dyn);
  const double w = i > 0 ? lyd / dxw : 0, e = i < lx - 1 ? lyd / dxe : 0;
  const double s = j > 0 ? lxd / dys : 0, n = j < ly - 1 ? lxd / dyn : 0;
  const int f = naFineIndex(lv, l, j, true) * nx0 + naFineIndex(lv, l, i, false);
  double d = __dadd_rn(__dadd_rn(__dadd_rn(w, e), s), n);
  d = __dadd_rn(__dadd_rn(d, __dmul_rn(gDx[f], lyd)), __dmul_rn(gDy[f], lxd));
  M.cw[k] = (float)w;
  M.ce[k] = (float)e;
  M.cs[k] = (float)s;
  M.cn[k] = (float)n;
  M.area[k] = (float)(lxd * lyd);
  M.diag0[k] = (float)d;
  if (l > 0)
    M.fixed[k] = fixed0[f];
}

// The distinct coefficient tuples of level blockIdx.y and each node's class
// (coefficientClasses on the device): a hash table of kNAClasses slots, each
// named by the node that claimed it first; tuples are compared bit for bit.
// Which slot a tuple gets depends on the order of the threads, its values do
// not.  More tuples than slots: *bad.
__global__ void naClassKernel(const __grid_constant__ NASet set, int *slots, int *bad) {
  const int l = blockIdx.y;
  const MGLevel &M = set.L[l];
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= M.nx * M.ny)
    return;
  auto tuple = [&](int q, uint32_t t[7]) {
    const float *f[6] = {M.cw, M.ce, M.cs, M.cn, M.area, M.diag0};
#pragma unroll
    for (int a = 0; a < 6; a++)
      t[a] = __float_as_uint(f[a][q]);
    t[6] = M.fixed[q] ? __float_as_uint(1.f) : 0u;
  };
  uint32_t t[7], o[7];
  tuple(k, t);
  uint32_t h = 2166136261u;
#pragma unroll
  for (int a = 0; a < 7; a++)
    h = (h ^ t[a] ^ (t[a] >> 15)) * 16777619u;
  h = (h ^ (h >> 13)) & (kNAClasses - 1);
  for (int probe = 0; probe < kNAClasses; probe++, h = (h + 1) & (kNAClasses - 1)) {
    int *slot = slots + l * kNAClasses + h;
    int r = *(volatile int *)slot;
    if (r < 0)
      r = atomicCAS(slot, -1, k);
    bool same = r < 0;
    if (same) { // claimed: the class's entry
      float *e = static_cast<float *>(M.clsTab) + 8 * h;
#pragma unroll
      for (int a = 0; a < 7; a++)
        e[a] = __uint_as_float(t[a]);
      e[7] = 0.f;
    } else {
      tuple(r, o);
      same = true;
#pragma unroll
      for (int a = 0; a < 7; a++)
        same = same && t[a] == o[a];
    }
    if (same) {
      M.cls[k] = (uint8_t)h;
      return;
    }
  }
  *bad = 1;
}

// 1-D transfer between level l (nf nodes) and level l + 1 (nc nodes) along one
// dimension: prolongation's lower coarse node and weight per fine node,
// restriction's (up to 3) fine nodes and weights per coarse node in ascending
// fine order, and the coarse -> fine injection map
// (blockIdx.y: level and, in its low bit, the dimension)
__global__ void naTransferKernel(const __grid_constant__ NALevels lv,
                                 const __grid_constant__ NASet set) {
  const int l = blockIdx.y >> 1;
  const bool ydim = blockIdx.y & 1;
  const MGLevel &M = set.L[l];
  int *pIdx = ydim ? M.pyIdx : M.pxIdx, *rIdx = ydim ? M.ryIdx : M.rxIdx;
  int *map = ydim ? M.mapY : M.mapX;
  float *pW = ydim ? M.pyW : M.pxW, *rW = ydim ? M.ryW : M.rxW;
  const int nf = ydim ? lv.ny[l] : lv.nx[l];
  const int nc = ydim ? lv.ny[l + 1] : lv.nx[l + 1];
  auto cmap = [&](int J) { return nf > 3 ? min(2 * J, nf - 1) : J; };
  auto X = [&](int i) { return naCoord(lv, l, i, ydim); };
  auto lower = [&](int i, int &I, float &w) {
    I = min(nf > 3 ? i / 2 : i, nc - 1);
    while (I + 1 < nc && cmap(I + 1) <= i)
      I++;
    while (I > 0 && cmap(I) > i)
      I--;
    if (cmap(I) == i || I + 1 >= nc)
      w = 1.f;
    else
      w = (float)((X(cmap(I + 1)) - X(i)) / (X(cmap(I + 1)) - X(cmap(I))));
  };
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nf) {
    int I;
    float w;
    lower(t, I, w);
    pIdx[t] = I;
    pW[t] = w;
  }
  if (t < nc) {
    map[t] = cmap(t);
    for (int q = 0; q < 3; q++) {
      rIdx[3 * t + q] = 0;
      rW[3 * t + q] = 0.f;
    }
    int cnt = 0;
    const int lo = t > 0 ? cmap(t - 1) : 0, hi = t + 1 < nc ? cmap(t + 1) : nf - 1;
    for (int i = lo; i <= hi && cnt < 3; i++) {
      int I;
      float w;
      lower(i, I, w);
      if (I == t && w > 0.f) {
        rIdx[3 * t + cnt] = i;
        rW[3 * t + cnt] = w;
        cnt++;
      } else if (I + 1 == t && w < 1.f) {
        rIdx[3 * t + cnt] = i;
        rW[3 * t + cnt] = 1.f - w;
        cnt++;
      }
    }
  }
}

} // namespace

// the array and its per-device address
static __device__ __align__(256) unsigned char g_poissonScratch[kNABytes];
static std::atomic<void *> g_poissonScratchAddr[kNAMaxDevices];

// The kernels of every form of the solve, loaded: the runtime loads a kernel at its
// first use, into device memory, and which form a call takes depends on its grid.  So
// the first call on a device loads them all, and no later one takes memory.
template <class... K> static int32_t loadKernels(K... k) {
  cudaFuncAttributes fa;
  cudaError_t e = cudaSuccess;
  ((e = e == cudaSuccess ? cudaFuncGetAttributes(&fa, k) : e), ...);
  EMCG_CUDA(e);
  return EMCG_OK;
}
static int32_t loadSolveKernels() {
  return loadKernels(naFineSetupKernel, naLevelSetupKernel, naTransferKernel, naClassKernel,
                     expTableKernel, resetBCKernel, nonlinResidualKernel<float>,
                     smoothKernel<float>, restrictKernel<float>, prolongKernel<float>,
                     coarseSolveKernel<float>, updatePotKernel<float>,
                     poissonClusterKernel<float, false, false>,
                     poissonClusterKernel<float, false, true>,
                     poissonClusterKernel<float, true, false>,
                     poissonClusterKernel<float, true, true>);
}

static int32_t poissonScratchAddress(unsigned char **out) {
  int dev = -1;
  EMCG_CUDA(cudaGetDevice(&dev));
  EMCG_CHECK_ARG(dev >= 0 && dev < kNAMaxDevices, "device %d is beyond the %d devices supported",
                 dev, kNAMaxDevices);
  void *p = g_poissonScratchAddr[dev].load(std::memory_order_acquire);
  if (!p) {
    cudaError_t e = cudaGetSymbolAddress(&p, g_poissonScratch);
    if (e != cudaSuccess || !p) {
      setError("cudaGetSymbolAddress of the Poisson scratch array failed on device %d: %s", dev,
               cudaGetErrorString(e));
      return EMCG_ERR_CUDA;
    }
    EMCG_TRY(loadSolveKernels());
    g_poissonScratchAddr[dev].store(p, std::memory_order_release);
  }
  *out = static_cast<unsigned char *>(p);
  return EMCG_OK;
}

} // namespace emcg

// the form of the thread's last solve (emcg_poisson_noalloc_form)
static thread_local int32_t g_noallocForm[3] = {};

extern "C" int32_t emcg_poisson_noalloc_form(int32_t *ctas, int32_t *tail_level,
                                             int32_t *tail_ctas) {
  int32_t *const out[3] = {ctas, tail_level, tail_ctas};
  for (int k = 0; k < 3; k++)
    if (out[k])
      *out[k] = g_noallocForm[k];
  return EMCG_OK;
}

extern "C" int32_t emcg_poisson_solve_noalloc(const emcg_device_desc *dv, double *d_pot,
                                              const double *d_conc, int32_t reset_bc,
                                              int32_t smooth, double rtol, int32_t max_cycles,
                                              void *cuda_stream, double *rel_residual,
                                              int32_t *cycles) {
  using namespace emcg;
  EMCG_CHECK_ARG(dv && d_pot, "device description and potential are required");
  const int nx = dv->nx, ny = dv->ny;
  EMCG_CHECK_ARG(nx >= 3 && ny >= 3, "grid must have at least 3 x 3 nodes (got %d x %d)", nx, ny);
  EMCG_CHECK_ARG(nx <= kNAMaxDim && ny <= kNAMaxDim && (int64_t)nx * ny <= kNAMaxNodes,
                 "grid %d x %d exceeds the no-allocation Poisson limit of %d nodes and %d per "
                 "dimension",
                 nx, ny, kNAMaxNodes, kNAMaxDim);
  EMCG_CHECK_ARG(dv->n_contacts >= 0 && dv->n_contacts <= kNAMaxContacts,
                 "%d contacts exceed the no-allocation Poisson limit of %d", dv->n_contacts,
                 kNAMaxContacts);
  EMCG_CHECK_ARG(dv->doping && dv->boundary_contact[0] && dv->boundary_contact[1] &&
                     dv->boundary_contact[2] && dv->boundary_contact[3],
                 "doping and boundary contact arrays are required");
  EMCG_CHECK_ARG(dv->n_contacts == 0 ||
                     (dv->contact_type && dv->contact_voltage && dv->contact_param),
                 "contact arrays are required");
  EMCG_CHECK_ARG(dv->hx > 0 && dv->hy > 0 && dv->temperature > 0 && dv->ni > 0 && dv->eps_r > 0,
                 "spacing, temperature, ni and eps_r must be positive");
  EMCG_CHECK_ARG(rtol > 0 && max_cycles >= 0 && smooth >= 0, "bad Poisson settings");
  for (int c = 0; c < dv->n_contacts; c++)
    EMCG_CHECK_ARG(dv->contact_type[c] == EMCG_CONTACT_OHMIC ||
                       dv->contact_type[c] == EMCG_CONTACT_GATE,
                   "contact %d: only ohmic and gate contacts are supported", c);
  for (int b = 0; b < 4; b++)
    for (int k = 0; k < (b < 2 ? ny : nx); k++)
      EMCG_CHECK_ARG(dv->boundary_contact[b][k] >= -1 &&
                         dv->boundary_contact[b][k] < dv->n_contacts,
                     "boundary %d, node %d: contact index %d out of range", b, k,
                     dv->boundary_contact[b][k]);
  // level shapes and their scratch footprint, checked before anything is written
  NALevels lv;
  lv.n = 0;
  size_t nodes = 0, oneD = 0;
  for (int l = 0, lx = nx, ly = ny; l < kNAMaxLevels; l++) {
    lv.nx[l] = lx;
    lv.ny[l] = ly;
    lv.n = l + 1;
    nodes += (size_t)lx * ly;
    const int cx = lx > 3 ? lx / 2 + 1 : lx, cy = ly > 3 ? ly / 2 + 1 : ly;
    if (cx == lx && cy == ly)
      break;
    oneD += (size_t)lx + ly + 4 * (size_t)cx + 4 * (size_t)cy;
    lx = cx;
    ly = cy;
  }
  EMCG_CHECK_ARG(nodes <= (size_t)kNALevelNodes && oneD <= (size_t)kNA1D,
                 "grid %d x %d: multigrid hierarchy exceeds the no-allocation scratch", nx, ny);
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  unsigned char *S = nullptr;
  EMCG_TRY(poissonScratchAddress(&S));
  const int n = nx * ny;
  // normalisation (include/emcDevice.hpp:87, emcSORSolver.hpp:330-368)
  const double Vt = kKB / kQ * dv->temperature;
  const double Ld = std::sqrt(kEPS0 * dv->eps_r * Vt / kQ / dv->ni);
  lv.h0 = dv->hx / Ld;
  lv.h1 = dv->hy / Ld;
  NAContacts ct;
  for (int c = 0; c < dv->n_contacts; c++) {
    ct.volt[c] = dv->contact_voltage[c] / Vt;
    ct.gF[c] = ct.barrier[c] = 0;
    if (dv->contact_type[c] == EMCG_CONTACT_GATE) {
      const double gamma = dv->contact_param[3 * c + 0] / dv->eps_r;
      const double tox = dv->contact_param[3 * c + 1] / Ld;
      ct.gF[c] = 2 * gamma / tox;
      ct.barrier[c] = dv->contact_param[3 * c + 2] / Vt;
    }
  }
  double *doping = (double *)(S + kOffDoping), *C = (double *)(S + kOffC);
  double *gSum = (double *)(S + kOffGSum), *gVeq = (double *)(S + kOffGVeq);
  double *gVne = (double *)(S + kOffGVne), *gDx = (double *)(S + kOffGDx);
  double *gDy = (double *)(S + kOffGDy), *resEq = (double *)(S + kOffResEq);
  double *resNe = (double *)(S + kOffResNe), *stats = (double *)(S + kOffStats);
  float *levF = (float *)(S + kOffLevelF), *trF = (float *)(S + kOffTransF);
  int *trI = (int *)(S + kOffTransI);
  int8_t *bnd = (int8_t *)(S + kOffBnd);
  uint8_t *resMask = S + kOffResMask, *fixedAll = S + kOffFixed;
  EMCG_CUDA(cudaMemcpyAsync(doping, dv->doping, sizeof(double) * n, cudaMemcpyHostToDevice, st));
  // the boundaries' contacts and the contact types behind them, in one copy
  int8_t hBnd[kNAMaxEdge];
  int8_t *put = hBnd;
  for (int b = 0; b < 4; b++)
    for (int k = 0; k < (b < 2 ? ny : nx); k++)
      *put++ = (int8_t)dv->boundary_contact[b][k];
  const int8_t *ctype = bnd + (put - hBnd);
  for (int c = 0; c < dv->n_contacts; c++)
    *put++ = (int8_t)dv->contact_type[c];
  EMCG_CUDA(cudaMemcpyAsync(bnd, hBnd, (size_t)(put - hBnd), cudaMemcpyHostToDevice, st));
  const double hF0 = lv.h1 / lv.h0, hF1 = lv.h0 / lv.h1;
  double hP = 1.;
  hP = hP * lv.h0;
  hP = hP * lv.h1;
  naFineSetupKernel<<<(n + kBlock - 1) / kBlock, kBlock, 0, st>>>(
      nx, ny, dv->ni, hF0, hF1, lv.h0, lv.h1, ct, doping, bnd, ctype, C, gSum, gVeq, gVne, gDx,
      gDy, resMask, resEq, resNe, fixedAll);
  EMCG_CUDA(cudaGetLastError());
  // carve the levels out of the scratch and build them
  NASet set;
  MGLevel *lev = set.L;
  size_t fo = 0, uo = 0, to = 0;
  float *tab = (float *)(S + kOffTab);
  int *slots = (int *)(S + kOffSlot), *bad = (int *)(S + kOffBad);
  double *expT = (double *)(S + kOffExp);
  for (int l = 0; l < lv.n; l++) {
    MGLevel &M = lev[l];
    std::memset(&M, 0, sizeof(M));
    M.nx = lv.nx[l];
    M.ny = lv.ny[l];
    const size_t m = (size_t)M.nx * M.ny;
    float **arr[9] = {&M.cw, &M.ce, &M.cs, &M.cn, &M.area, &M.diag0, &M.d, &M.r, &M.rho};
    for (int a = 0; a < 9; a++) {
      *arr[a] = levF + fo;
      fo += m;
    }
    M.fixed = fixedAll + uo;
    M.cls = S + kOffCls + uo;
    uo += m;
    M.clsTab = tab + 8 * kNAClasses * l;
    M.nCls = kNAClasses;
    if (l + 1 < lv.n) {
      const int ncx = lv.nx[l + 1], ncy = lv.ny[l + 1];
      M.pxIdx = trI + to;
      M.pxW = trF + to;
      to += M.nx;
      M.pyIdx = trI + to;
      M.pyW = trF + to;
      to += M.ny;
      M.rxIdx = trI + to;
      M.rxW = trF + to;
      to += 3 * (size_t)ncx;
      M.ryIdx = trI + to;
      M.ryW = trF + to;
      to += 3 * (size_t)ncy;
      M.mapX = trI + to;
      to += ncx;
      M.mapY = trI + to;
      to += ncy;
    }
  }
  // (slots to -1, the overflow flag to 0, the statistics to 0)
  EMCG_CUDA(cudaMemsetAsync(slots, 0xff, sizeof(int) * kNAMaxLevels * kNAClasses, st));
  EMCG_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), st));
  const int nodeBlocks = (n + kBlock - 1) / kBlock;
  naLevelSetupKernel<<<dim3(nodeBlocks, lv.n), kBlock, 0, st>>>(lv, set, gDx, gDy, fixedAll, nx);
  EMCG_CUDA(cudaGetLastError());
  if (lv.n > 1) {
    naTransferKernel<<<dim3((std::max(nx, ny) + kBlock - 1) / kBlock, 2 * (lv.n - 1)), kBlock, 0,
                       st>>>(lv, set);
    EMCG_CUDA(cudaGetLastError());
  }
  naClassKernel<<<dim3(nodeBlocks, lv.n), kBlock, 0, st>>>(set, slots, bad);
  expTableKernel<<<1, kExpTab, 0, st>>>(expT);
  EMCG_CUDA(cudaGetLastError());
  // Newton / defect correction: the loop of the allocating solver (float MG)
  const int grid = (n + kBlock - 1) / kBlock;
  if (reset_bc) {
    resetBCKernel<<<grid, kBlock, 0, st>>>(d_pot, resMask, d_conc ? resNe : resEq, n);
    EMCG_CUDA(cudaGetLastError());
  }
  const int pre = smooth > 0 ? smooth : 3, post = pre, coarseSweeps = 16;
  const MGSet mg = {lev, lv.n, pre, post, coarseSweeps, kNAVcyclesPerNewton, kNATwoCycleRel};
  LevelK<float> K0 = levelK<float>(lev[0]);
  double h_stats[3] = {0, 0, 0};
  double rel = INFINITY;
  int it = 0;
  double scale = 0.;
  // the whole solve in one cluster launch where the grid fits (201 x 101: 4.28 ms
  // with one launch per phase, 0.69 ms so)
  const ClusterFit fit = clusterFit<float, false>(mg, 0, 1);
  bool done = false;
  if (fit.size) {
    size_t bytes = 0;
    const CMG<float> M = clusterDesc<float>(mg, fit.size, &bytes, fit.even);
    cudaLaunchAttribute at;
    cudaLaunchConfig_t cfg = clusterConfig<float>(fit.size, bytes, st, &at);
    EMCG_CUDA(cudaLaunchKernelEx(&cfg, clusterKernel<float, false>(M), M, d_pot, d_conc,
                                 (const double *)C, (const double *)gSum,
                                 (const double *)(d_conc ? gVne : gVeq), hF0, hF1, hP, rtol,
                                 (int)max_cycles, 0., (const double *)expT, stats,
                                 (const float *)nullptr, (const float *)nullptr, (float *)nullptr,
                                 (const int *)bad));
    EMCG_CUDA(cudaMemcpyAsync(h_stats, stats, 3 * sizeof(double), cudaMemcpyDeviceToHost, st));
    EMCG_CUDA(cudaStreamSynchronize(st));
    done = h_stats[2] >= 0.; // a table overflowed: one launch per phase
    if (done) {
      rel = h_stats[0];
      it = (int)h_stats[1];
    }
  }
  MGTail tail;
  if (!done && !fit.size) {
    ClusterFit t;
    int h_bad = 0;
    EMCG_CUDA(cudaMemcpyAsync(&h_bad, bad, sizeof(int), cudaMemcpyDeviceToHost, st));
    EMCG_CUDA(cudaStreamSynchronize(st));
    if (!h_bad) {
      tailPlan<float>(mg, 0, tail.level, t);
      tail.size = t.size;
      tail.even = t.even;
    }
  }
  g_noallocForm[0] = done ? fit.size : 0;
  g_noallocForm[1] = tail.level;
  g_noallocForm[2] = tail.level ? tail.size : 0;
  for (; !done && it <= max_cycles; it++) {
    // the residual maxima accumulate by atomic max and must start at zero
    EMCG_CUDA(cudaMemsetAsync(stats, 0, 4 * sizeof(double), st));
    nonlinResidualKernel<float><<<grid, kBlock, 0, st>>>(
        d_pot, d_conc, C, lev[0].fixed, gSum, d_conc ? gVne : gVeq, nx, ny, hF0, hF1, hP, K0.r,
        K0.rho, K0.d, stats, it == 0);
    EMCG_CUDA(cudaGetLastError());
    EMCG_CUDA(cudaMemcpyAsync(h_stats, stats, 2 * sizeof(double), cudaMemcpyDeviceToHost, st));
    EMCG_CUDA(cudaStreamSynchronize(st));
    if (it == 0)
      scale = h_stats[1];
    rel = scale > 0 ? h_stats[0] / scale : h_stats[0];
    if (rel <= rtol || it == max_cycles || !std::isfinite(rel))
      break;
    const int nv = rel < kNATwoCycleRel ? kNAVcyclesPerNewton : 1;
    for (int k = 0; k < nv; k++)
      vcycle<float>(mg, 0, tail, st);
    EMCG_CUDA(cudaGetLastError());
    updatePotKernel<float><<<grid, kBlock, 0, st>>>(d_pot, K0.d, lev[0].fixed, n, stats);
    EMCG_CUDA(cudaGetLastError());
  }
  if (rel_residual)
    *rel_residual = rel;
  if (cycles)
    *cycles = it;
  if (!std::isfinite(rel)) {
    setError("Poisson: non-finite residual after %d Newton steps (NaN or Inf in the potential, "
             "the concentration or a correction)", it);
    return EMCG_ERR_NONCONVERGED;
  }
  if (!(rel <= rtol)) {
    setError("Poisson: relative residual %.3e after %d Newton steps (target %.1e)", rel, it, rtol);
    return EMCG_ERR_NONCONVERGED;
  }
  return EMCG_OK;
}
