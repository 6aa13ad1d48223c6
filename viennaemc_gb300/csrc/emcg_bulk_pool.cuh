// Pooled step kernel of the double engine (Philox draws): each warp owns a
// pool of electrons in shared memory and works on up to 32 of them at a time
// that all need the same thing.
//
// What bounds it: the double-precision pipe.  Each of an SM's four schedulers
// issues one double instruction of a warp in 64 clocks, however many lanes are
// active and however independent the instructions are (measured), so a branch
// taken by 4 of 32 lanes costs as much as one taken by all.  In a kernel whose
// warps carry 32 electrons step by step, a step of 1 fs holds an event for about
// every fourth electron: nearly every warp runs the event path, with a few
// lanes, in every step (about 350 double instructions per 32 particle-steps).
// Here the warp sorts its electrons by what they need next --
//   flight   fly to the end of the step or the next event;
//   select   draw the mechanism (most draws are self-scattering) and the new
//            free flight;
//   scatter  the final state of a real mechanism;
// -- and runs the kind of which 32 are ready, so the lanes of a pass are full.
// Electrons run ahead of each other by at most kPoolWindow steps; the energy
// and velocity of each (step, electron) wait in shared memory until every
// electron of the pool has passed the step, then eight lanes per step add them
// up (in double, one addition per electron and quantity, not five of a
// butterfly).  k stays in the ellipse frame of its subvalley and is rotated
// only by real scattering, as in the float engine's warp-asynchronous kernel.
// Measured, lockstep -> pools: 10,000 electrons x 100 steps 3.65 -> 1.01 ms a call
// with its read-back, 250,007 x 20 steps 4.00 -> 0.94 ms, 10^6 electrons 1.8e9
// -> 5.6e9 particle-steps/s, 92 double instructions per 32 particle-steps at 83 %
// of the pipe.  A window of 16 steps costs resident pools (4.6e9), one of 4 with
// 128 electrons per pool gains 4 % at 10^6 electrons and loses as much at 10^4.
// Integer instructions replace double ones where the result is the same bit for
// bit: comparisons of table entries, the draws' conversion, the energy level,
// rotations into frames along the device's axes.
#pragma once

#include "emcg_common.cuh"
#include "emcg_log.h"

namespace emcg {

constexpr int kPoolWindow = 8; // steps an electron may be ahead of the pool's slowest
constexpr int kPoolFold = 4;   // steps added up at a time, by eight lanes each
constexpr int kPoolFields = 13; // k, d, E, tau, gtau, in, x in shared memory
constexpr uint32_t kPoolMaxEvents = 1u << 16; // of one electron in one step

// an electron's kind word: PoolKind, its mechanism in bits 8 to 12, its events in the
// step above, and kPoolFar: its next flight is wrapped by itself (poolFarFlight)
enum PoolKind : uint32_t { kFlight = 0, kSelect = 1, kScatter = 2, kDone = 3 };
constexpr uint32_t kKindMask = 0xffu, kPoolEvent = 1u << 13, kPoolFar = 1u << 31;
static_assert(EMCG_MAX_MECH <= 32 && kPoolMaxEvents < (1u << 18), "the kind word's fields");

template <int G> struct PoolShape {
  static constexpr int P = 32 * G;
  // a row of the window: 8 doubles of padding put two rows that the sum reads
  // together on different banks
  static constexpr int PW = P + 8;
};

template <int G> __host__ __device__ constexpr size_t poolSmemBytes(bool one) {
  constexpr size_t P = PoolShape<G>::P, PW = PoolShape<G>::PW;
  return sizeof(double) * 2 * kPoolWindow * PW + (one ? 0 : kPoolWindow * P) +
         (G > 1 ? sizeof(double) * kPoolFields * P + 4 * 4 * P + 32 : 0);
}

// One Philox block and the draws' log out of line: the code of a pass is run a
// few times per launch in short launches, and its instruction fetches cost
// more than the calls
__device__ __noinline__ uint4 poolPhilox(uint32_t pid, uint32_t step, uint32_t call,
                                         uint32_t stream, uint32_t k0, uint32_t k1) {
  uint32_t o[4];
  philox4x32_10(pid, step, call, stream, k0, k1, o);
  return make_uint4(o[0], o[1], o[2], o[3]);
}
__device__ __noinline__ double poolLog(double x, const double *tab) { return logTab(x, tab); }

// The draws of one electron in one step: word i of its Philox stream (the
// counter's call i / 2, or i / 4 for 32-bit draws), so only the count of words
// consumed is kept between passes.
struct PoolDraws {
  uint32_t pid, step, stream, k0, k1;
  uint32_t i, have;
  uint4 o;
  bool f32;
  __device__ __forceinline__ PoolDraws(const EnsK<double> &EK, uint32_t pid_, uint32_t step_,
                                       uint32_t words)
      : pid(pid_), step(step_), stream(EK.stream), k0(EK.key0), k1(EK.key1), i(words),
        have(0xffffffffu), f32(EK.floatDraws != 0) {}
  __device__ __forceinline__ void load(uint32_t call) {
    if (call != have) {
      o = poolPhilox(pid, step, call, stream, k0, k1);
      have = call;
    }
  }
  __device__ __forceinline__ uint64_t word() {
    load(i >> 1);
    const uint64_t w = i & 1 ? (uint64_t)o.z | ((uint64_t)o.w << 32)
                             : (uint64_t)o.x | ((uint64_t)o.y << 32);
    i++;
    return w;
  }
  __device__ __forceinline__ uint32_t word32() {
    load(i >> 2);
    const uint32_t w = (i & 3) == 0 ? o.x : (i & 3) == 1 ? o.y : (i & 3) == 2 ? o.z : o.w;
    i++;
    return w;
  }
  __device__ __forceinline__ uint32_t pick(uint32_t n) {
    if (f32)
      return __umulhi(word32(), n);
    const uint64_t w = word();
    return (n & (n - 1)) == 0 ? (uint32_t)w & (n - 1) : (uint32_t)(w % (uint64_t)n);
  }
  __device__ __forceinline__ double u01() {
    return f32 ? (double)((float)(word32() >> 8) * 0x1p-24f) : canonicalBits(word());
  }
  __device__ __forceinline__ double ulog() {
    if (f32)
      return (double)fmaf((float)(word32() >> 8) * 0x1p-24f, 1.f - 1e-6f, 1e-6f);
    return __dadd_rn(__dmul_rn(canonicalBits(word()), 1. - 1e-6), 1e-6);
  }
};

// one electron of a pool
struct PoolEl {
  double k[3], d[3], x[3]; // ellipse-frame k, its displacement not yet in x, position
  double E, tau, gtau, in; // in: time spent inside the step
  int step;
  uint32_t words, meta, kind; // draws consumed in the step; the kind word above
};

// The summed ellipse-frame displacement into the device frame and the periodic
// box, as flushPos of the float engine: flights of less than half a box from a position
// inside it, for which this is the reference's rule (basicBulkParticleHandler.hpp:
// 600-613: one box length added or taken after each flight).  kPoolFar: none is summed.
__device__ __forceinline__ void poolFlush(const ValleyK<double> &V, int sub, const double box[3],
                                          PoolEl &p) {
  if (p.kind & kPoolFar)
    return;
  double d[3], dd[3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    d[i] = p.d[i] * V.vogt[i];
    p.d[i] = 0.0;
  }
  rotate<true>(V, sub, d, dd);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    double c = p.x[i] + dd[i];
    if (negativeD(c) || belowD(box[i], c))
      c -= box[i] * floor(c / box[i]);
    p.x[i] = c;
  }
}

// outside the box
__device__ __forceinline__ bool poolOutside(const double *box, double x, double y, double z) {
  return negativeD(x) || belowD(box[0], x) || negativeD(y) || belowD(box[1], y) ||
         negativeD(z) || belowD(box[2], z);
}
// A flight that may be longer than half a box, or that starts outside it: the earlier
// flights' displacement d into the position (unless far: there is none), then this
// one's, i, with the reference's rule.  A call, by values: it is rare, and the flights'
// sums stay in registers.
struct PoolFarPos {
  double x[3];
  bool out;
};
__device__ __noinline__ PoolFarPos poolFarFlight(const ValleyK<double> *V, int sub,
                                                 const double *box, bool far, double d0,
                                                 double d1, double d2, double i0, double i1,
                                                 double i2, double x0, double x1, double x2) {
  const double d[2][3] = {{d0 * V->vogt[0], d1 * V->vogt[1], d2 * V->vogt[2]},
                          {i0 * V->vogt[0], i1 * V->vogt[1], i2 * V->vogt[2]}};
  double s[3], t[3];
  rotate<true>(*V, sub, d[0], s);
  rotate<true>(*V, sub, d[1], t);
  const double x[3] = {x0, x1, x2};
  PoolFarPos o;
  for (int i = 0; i < 3; i++) {
    double c = x[i];
    if (!far) {
      c += s[i];
      if (negativeD(c) || belowD(box[i], c))
        c -= box[i] * floor(c / box[i]);
    }
    c += t[i];
    if (negativeD(c))
      c += box[i];
    else if (belowD(box[i], c))
      c -= box[i];
    o.x[i] = c;
  }
  o.out = poolOutside(box, o.x[0], o.x[1], o.x[2]);
  return o;
}

// the grain timer ran out (basicBulkParticleHandler.hpp:215-219)
__device__ __forceinline__ void poolGrain(const ModelK<double> &M, const EnsK<double> &EK,
                                       uint32_t pid, uint32_t step, PoolEl &p) {
  PoolDraws rng(EK, pid, step, p.words);
  if (M.grain) {
    const double *R = M.v[p.meta & 0xff].rot[(p.meta >> 8) & 0xff];
    double k[3];
    toDev(R, p.k[0], p.k[1], p.k[2], k);
    grainScatter(M, k, rng);
    toEcs(R, k[0], k[1], k[2], p.k);
  }
  p.gtau = -poolLog(rng.ulog(), M.logT) * M.grainTau;
}

struct PoolValley { // a valley's constants of the free flight
  double cE, alpha2, cX; // hbar^2 / (mc q), 2 alpha, hbar / mc
  uint32_t farK2;        // EnsK::farK2
};

// A free flight of p (drift(), include/emcParticleDrift.hpp:11-36, in the ellipse
// frame) to the end of its step or its next event; true at the end of the step,
// vd then the velocity along the field.  x(i): the position, where it is kept.
template <class X>
__device__ __forceinline__ bool poolFlight(const PoolValley &V, const EnsK<double> &EK,
                                           const ModelK<double> &M, int valley, int sub,
                                           uint32_t pid, uint32_t step0, PoolEl &p, X x,
                                           double &vd) {
  const double *fv = EK.fv[valley][sub];
  const double rem = EK.dt - p.in;
  const bool ev = belowD(p.tau, rem);
  const double t = ev ? p.tau : rem;
  double kO[3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    kO[i] = p.k[i];
    p.k[i] = fma(fv[i], t, kO[i]);
  }
  double rs;
  const double k2 = fma(p.k[2], p.k[2], fma(p.k[1], p.k[1], p.k[0] * p.k[0]));
  p.E = energyRoot(V.cE, V.alpha2, k2, rs);
  const double vh = V.cX * (0.5 * rs); // hbar / (2 mc (1 + 2 alpha E))
  const double c = vh * t;
  const bool big = (uint32_t)__double2hiint(k2) >= V.farK2;
  if (big || (p.kind & kPoolFar)) {
    const PoolFarPos o = poolFarFlight(
        &M.v[valley], sub, EK.box, p.kind & kPoolFar, p.d[0], p.d[1], p.d[2],
        (p.k[0] + kO[0]) * c, (p.k[1] + kO[1]) * c, (p.k[2] + kO[2]) * c, x(0), x(1), x(2));
#pragma unroll
    for (int i = 0; i < 3; i++) {
      x(i) = o.x[i];
      p.d[i] = 0.0;
    }
    p.kind = (p.kind & ~kPoolFar) | (big || o.out ? kPoolFar : 0u);
  } else {
#pragma unroll
    for (int i = 0; i < 3; i++)
      p.d[i] = fma(p.k[i] + kO[i], c, p.d[i]);
  }
  if (ev) {
    p.in += t;
    p.kind |= kSelect; // (from kFlight)
    return false;
  }
  p.tau -= t;
  p.in = 0.0;
  p.gtau -= EK.dt;
  if (notPositiveD(p.gtau))
    poolGrain(M, EK, pid, step0 + (uint32_t)p.step, p);
  const double *gd = EK.g[valley][sub];
  const double gk = fma(gd[2], p.k[2], fma(gd[1], p.k[1], gd[0] * p.k[0]));
  vd = vh * (gk + gk);
  p.step++;
  p.words = 0;
  p.kind &= kPoolFar; // kFlight, no events
  return true;
}

// The event of p: the mechanism (scatterParticle, include/emcScatterHandler.hpp:
// 148-170) and the new free flight.  The flight's draw follows those of the final
// state: a mechanism's draws are counted here and taken in poolScatter.
template <bool kOne>
__device__ __forceinline__ int poolSelect(const EnsK<double> &EK, const ModelK<double> &M,
                                          uint32_t pid, uint32_t step0, PoolEl &p) {
  PoolDraws rng(EK, pid, step0 + (uint32_t)p.step, p.words);
  int valley = kOne ? 0 : (int)(p.meta & 0xff);
  const int region = p.meta >> 16;
  const int ts = M.tsIndex[valley][region];
  const uint32_t far = p.kind & kPoolFar, events = (p.kind & ~kPoolFar) / kPoolEvent;
  if (events >= kPoolMaxEvents)
    return EMCG_ERR_TIMEOUT;
  if (ts < 0)
    return EMCG_ERR_OUT_OF_TABLE;
  const int nT = M.tsN[ts];
  p.kind = far | (events + 1) * kPoolEvent; // kFlight
  if (nT > 0) {
    const long long rnd = __double_as_longlong(rng.u01());
    const double *row =
        M.tables + M.tsOff[ts] + (int64_t)levelFast(p.E, M.dE, M.invdE, M.nLevels) * nT;
    // non-negative doubles compare like their bit patterns
    if (rnd <= __double_as_longlong(ldg(row + nT - 1))) {
      int t = 0;
#pragma unroll 4
      for (int q = 0; q < nT; q++)
        t += __double_as_longlong(ldg(row + q)) <= rnd ? 1 : 0;
      if (t < nT) {
        const int mi = M.tsMech[ts][t];
        const MechK<double> &me = M.m[mi];
        p.kind |= kScatter | (uint32_t)mi << 8;
        p.words = rng.i;
        valley = kOne ? 0 : me.finalValley;
        // a direction takes two draws, an intervalley event its subvalley's too
        rng.i += me.kind == EMCG_MECH_ACOUSTIC || me.kind == EMCG_MECH_COULOMB ? 2 : 3;
      }
    }
  }
  p.tau = -poolLog(rng.ulog(), M.logT) * tauOf(M, valley, region);
  if ((p.kind & kKindMask) == kFlight)
    p.words = rng.i;
  return 0;
}

// The final state of p's mechanism (applyMechanism).
template <bool kOne>
__device__ __forceinline__ void poolScatter(const EnsK<double> &EK, const ModelK<double> &M,
                                            uint32_t pid, uint32_t step0, PoolEl &p) {
  PoolDraws rng(EK, pid, step0 + (uint32_t)p.step, p.words);
  const MechK<double> &me = M.m[(p.kind >> 8) & 31u];
  int valley = kOne ? 0 : (int)(p.meta & 0xff), sub = (p.meta >> 8) & 0xff;
  const int region = p.meta >> 16;
  double kd[3];
  bool big = false; // (an elastic mechanism keeps |k|)
  poolFlush(M.v[valley], sub, EK.box, p);
  if (me.kind == EMCG_MECH_COULOMB) {
    toDev(M.v[valley].rot[sub], p.k[0], p.k[1], p.k[2], kd);
    applyMechanism(M, me, kd, p.E, valley, sub, region, rng);
  } else {
    double n2; // the new |k|^2; elastic: |k| is the same in both frames
    if (me.kind == EMCG_MECH_ACOUSTIC) {
      n2 = p.k[0] * p.k[0] + p.k[1] * p.k[1] + p.k[2] * p.k[2];
    } else {
      if (!kOne)
        valley = me.finalValley;
      sub = me.finalSub[sub][rng.pick((uint32_t)me.nF)];
      p.E += me.shift;
      p.meta = packMeta(valley, sub, region);
      const double cK = M.v[valley].cK;
      n2 = cK * cK * gammaOf(M.v[valley], p.E);
      big = (uint32_t)__double2hiint(n2) >= EK.farK2[valley];
    }
    const double nk = sqrtD(n2);
    const double ct = 1.0 - 2.0 * rng.u01(), r1 = rng.u01();
    double sn, cs;
    sincospi(2.0 * r1, &sn, &cs);
    const double ns = nk * sqrtD(1.0 - ct * ct);
    kd[0] = ns * cs;
    kd[1] = ns * sn;
    kd[2] = nk * ct;
  }
  rotate<false>(M.v[valley], sub, kd, p.k);
  p.words = rng.i + 1; // the free flight's draw is taken
  p.kind &= ~(kPoolEvent - 1); // kFlight
  if (big)
    p.kind |= kPoolFar;
}

// G: pools of up to 32 G electrons, one warp per block and pool; kOne: every
// ensemble of the launch has one valley.  With G = 1 each lane keeps its
// electron in registers.
template <int G, bool kOne>
__global__ void __launch_bounds__(32)
    bulkStepPoolKernel(StateK<double> st, const ModelK<double> *__restrict__ models,
                       const EnsK<double> *__restrict__ ens, const Tile *__restrict__ tiles,
                       int nSteps, uint32_t step0, int nVmax, double *__restrict__ obs,
                       int *__restrict__ err) {
  constexpr int P = PoolShape<G>::P, PW = PoolShape<G>::PW, W = kPoolWindow;
  constexpr bool kReg = G == 1;
  extern __shared__ __align__(16) double poolSmem[];
  double *wE = poolSmem, *wD = wE + W * PW;               // [W][PW]
  double *f = wD + W * PW;                                // [kPoolFields][P], G > 1
  int *stp = reinterpret_cast<int *>(f + kPoolFields * P); // the step an electron is in
  uint32_t *words = reinterpret_cast<uint32_t *>(stp + P);
  uint32_t *meta = words + P, *kind = meta + P;
  uint8_t *list = reinterpret_cast<uint8_t *>(kind + P); // the electrons of a pass
  uint8_t *wV = kReg ? reinterpret_cast<uint8_t *>(f) : list + 32; // [W][P], several valleys
  const int lane = threadIdx.x;
  const Tile tl = tiles[blockIdx.x];
  const EnsK<double> &EK = ens[tl.ens];
  const ModelK<double> &M = models[EK.model];
  const int n = (int)(tl.end - tl.begin);
  const int nV = kOne ? 1 : EK.nV;
  const int Q = nVmax * 3;
  const uint32_t pid0 = (uint32_t)(tl.begin - EK.begin);
  // the one valley's constants, in registers
  const PoolValley one{M.v[0].cE, 2.0 * M.v[0].alpha, M.v[0].cX, EK.farK2[0]};
  int myErr = 0;

  PoolEl p;
  auto get = [&](int j, int from, int to) { // fields [from, to) of electron j
    double *const q[kPoolFields] = {&p.k[0], &p.k[1], &p.k[2], &p.d[0], &p.d[1], &p.d[2], &p.E,
                                    &p.tau,  &p.gtau, &p.in,   &p.x[0], &p.x[1], &p.x[2]};
    for (int i = from; i < to; i++)
      *q[i] = f[i * P + j];
  };
  auto put = [&](int j, int from, int to) {
    const double q[kPoolFields] = {p.k[0], p.k[1], p.k[2], p.d[0], p.d[1], p.d[2], p.E,
                                   p.tau,  p.gtau, p.in,   p.x[0], p.x[1], p.x[2]};
    for (int i = from; i < to; i++)
      f[i * P + j] = q[i];
  };
  p.kind = kDone;
  p.step = nSteps;
  for (int j = lane; j < P; j += 32) {
    p.kind = kDone;
    p.step = nSteps;
    p.words = 0;
    if (j < n) {
      const int64_t gi = tl.begin + j;
      p.meta = st.meta[gi];
      const double kd[3] = {st.kx[gi], st.ky[gi], st.kz[gi]};
      rotate<false>(M.v[p.meta & 0xff], (p.meta >> 8) & 0xff, kd, p.k);
      p.x[0] = st.px[gi];
      p.x[1] = st.py[gi];
      p.x[2] = st.pz[gi];
      p.E = st.E[gi];
      p.tau = st.tau[gi];
      p.gtau = st.gtau[gi];
      p.d[0] = p.d[1] = p.d[2] = p.in = 0.0;
      // (a negative timer of the caller's may be longer than a step)
      const double k2 = fma(p.k[2], p.k[2], fma(p.k[1], p.k[1], p.k[0] * p.k[0]));
      p.kind = (uint32_t)__double2hiint(k2) >= EK.farK2[p.meta & 0xff] ||
                       __double2hiint(p.tau) < 0 || poolOutside(EK.box, p.x[0], p.x[1], p.x[2])
                   ? kPoolFar
                   : 0u; // kFlight
      p.step = 0;
      if (!kReg)
        put(j, 0, kPoolFields);
    }
    if (!kReg) {
      stp[j] = p.step;
      words[j] = 0;
      meta[j] = p.meta;
      kind[j] = p.kind;
    }
  }
  __syncwarp();

  double *obsE = obs + (size_t)tl.ens * nSteps * Q;
  const int idle = min(24, n / 2); // fewer ready electrons than this: sum what can be summed
  int flushed = 0;                 // steps added to the ensemble's sums
  while (true) {
    // what the pool's electrons need
    unsigned mF[G], mS[G], mR[G], mL[G];
    int nF = 0, nS = 0, nR = 0, sMin = nSteps;
    const int limit = min(nSteps, flushed + W);
#pragma unroll
    for (int g = 0; g < G; g++) {
      const int s = kReg ? p.step : stp[32 * g + lane];
      const uint32_t k = (kReg ? p.kind : kind[32 * g + lane]) & kKindMask;
      mF[g] = __ballot_sync(0xffffffffu, k == kFlight && s < limit);
      mS[g] = __ballot_sync(0xffffffffu, k == kSelect);
      mR[g] = __ballot_sync(0xffffffffu, k == kScatter);
      mL[g] = G > 1 ? __ballot_sync(0xffffffffu, s < flushed + W / 2) : 0u;
      nF += __popc(mF[g]);
      nS += __popc(mS[g]);
      nR += __popc(mR[g]);
      sMin = min(sMin, s);
    }
    sMin = __reduce_min_sync(0xffffffffu, sMin);
    const int ready = sMin - flushed;
    if (ready >= kPoolFold || (ready > 0 && (sMin == nSteps || max(nF, max(nS, nR)) < idle))) {
      __syncwarp(); // the rows are written
      const int rows = min(ready, kPoolFold);
      const int row = lane >> 3, q = lane & 7, s = flushed + row;
      const int slot = s & (W - 1);
      for (int v = 0; v < nV; v++) {
        double e = 0.0, d = 0.0;
        int c = 0;
        if (row < rows)
          for (int j = q; j < n; j += 8)
            if (kOne || wV[slot * P + j] == v) {
              e += wE[slot * PW + j];
              d += wD[slot * PW + j];
              c++;
            }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
          e += __shfl_xor_sync(0xffffffffu, e, o);
          d += __shfl_xor_sync(0xffffffffu, d, o);
          c += __shfl_xor_sync(0xffffffffu, c, o);
        }
        if (row < rows && q == 0) {
          double *o = obsE + (size_t)s * Q + v * 3;
          atomicAdd(o + 0, e);
          atomicAdd(o + 1, d);
          atomicAdd(o + 2, (double)c);
        }
      }
      __syncwarp(); // the rows are read: their slots may be written again
      flushed += rows;
      continue;
    }
    if (nF + nS + nR == 0)
      break;
    // the kind with a full pass ready, the later stages first; else flights
    // while they are twice as many as the others (measured against 1, 1.5 and
    // 2/3 times as many on 300 to 4e5 electrons: 10,000 electrons 1.46e9
    // particle-steps/s against 1.35, 1.43 and 1.32)
    const int pick = nR >= 32 ? kScatter
                     : nS >= 32 ? kSelect
                     : nF >= 32 || (nF >= 2 * nS && nF >= 2 * nR) ? kFlight
                     : nS >= nR ? kSelect
                                : kScatter;
    bool act;
    int j = lane;
    if (kReg) {
      act = ((pick == kFlight ? mF[0] : pick == kSelect ? mS[0] : mR[0]) >> lane) & 1u;
    } else {
      // the electrons of the pass: those at the pool's first steps before those
      // that are ahead, so that few run into the window's end
      int cnt = 0;
#pragma unroll
      for (int late = 0; late < 2; late++)
#pragma unroll
        for (int g = 0; g < G; g++) {
          const unsigned m = (pick == kFlight ? mF[g] : pick == kSelect ? mS[g] : mR[g]) &
                             (late ? ~mL[g] : mL[g]);
          const int rank = cnt + __popc(m & ((1u << lane) - 1u));
          if (((m >> lane) & 1u) && rank < 32)
            list[rank] = (uint8_t)(32 * g + lane);
          cnt += __popc(m);
        }
      __syncwarp();
      act = lane < cnt;
      j = act ? list[lane] : 0;
      if (act) {
        p.step = stp[j];
        p.words = words[j];
        p.meta = meta[j];
        p.kind = kind[j];
      }
    }
    const uint32_t pid = pid0 + (uint32_t)j;
    if (!act) {
    } else if (pick == kFlight) {
      if (!kReg)
        get(j, 0, 10);
      const int valley = kOne ? 0 : (int)(p.meta & 0xff), sub = (p.meta >> 8) & 0xff;
      const ValleyK<double> &VK = M.v[valley];
      const PoolValley V =
          kOne ? one : PoolValley{VK.cE, 2.0 * VK.alpha, VK.cX, EK.farK2[valley]};
      auto x = [&](int i) -> double & { return kReg ? p.x[i] : f[(10 + i) * P + j]; };
      const int slot = p.step & (W - 1);
      double vd;
      if (poolFlight(V, EK, M, valley, sub, pid, step0, p, x, vd)) {
        wE[slot * PW + j] = p.E;
        wD[slot * PW + j] = vd;
        if (!kOne)
          wV[slot * P + j] = (uint8_t)valley;
        if (p.step >= nSteps)
          p.kind |= kDone;
      }
      if (!kReg)
        put(j, 0, 10);
    } else if (pick == kSelect) {
      if (!kReg)
        p.E = f[6 * P + j];
      const int e = poolSelect<kOne>(EK, M, pid, step0, p);
      if (e) {
        myErr = e;
        p.kind = kDone;
        p.step = nSteps;
      } else if (!kReg) {
        f[7 * P + j] = p.tau;
      }
    } else {
      if (!kReg) {
        get(j, 0, 7);
        get(j, 10, 13);
      }
      poolScatter<kOne>(EK, M, pid, step0, p);
      if (!kReg) {
        put(j, 0, 7);
        put(j, 10, 13);
      }
    }
    if (!kReg) {
      if (act) {
        stp[j] = p.step;
        words[j] = p.words;
        meta[j] = p.meta;
        kind[j] = p.kind;
      }
      __syncwarp();
    }
  }

  for (int j = lane; j < n; j += 32) {
    const int64_t gi = tl.begin + j;
    if (!kReg) {
      get(j, 0, kPoolFields);
      p.meta = meta[j];
      p.kind = kind[j];
    }
    const ValleyK<double> &V = M.v[p.meta & 0xff];
    const int sub = (p.meta >> 8) & 0xff;
    poolFlush(V, sub, EK.box, p);
    double k[3];
    rotate<true>(V, sub, p.k, k);
    st.kx[gi] = k[0];
    st.ky[gi] = k[1];
    st.kz[gi] = k[2];
    st.px[gi] = p.x[0];
    st.py[gi] = p.x[1];
    st.pz[gi] = p.x[2];
    st.E[gi] = p.E;
    st.tau[gi] = p.tau;
    st.gtau[gi] = p.gtau;
    st.meta[gi] = p.meta;
  }
  if (myErr)
    atomicCAS(err, 0, myErr);
}

} // namespace emcg
