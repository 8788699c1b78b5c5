// Direct-space pair kernel and force finalisation (sm_100a).
//
// Counterpart of getforce_nbdirect_kernel (src/nbdirect/nbdirect.cu:87-490)
// plus recull_blocks (src/domdec/recull.cu:41-122) and unpack_forces
// (src/domdec/assign_blocks.cu:444-468), redesigned for Blackwell SIMT:
//
//  * Work item = one i-block x up to 32 candidate j-tiles (the list rebuild
//    splits each block's candidates into items, work_split.h).  A warp
//    recull-tests its candidates at rCut with the fresh AABBs (one lane per
//    candidate, ballot), then walks the surviving tiles; the persistent warps
//    pull items from a counter, longest first once a launch has measured
//    their cycles (k_order).
//  * The j atoms of the surviving tiles that can reach the i block are queued
//    per warp in shared memory and evaluated in rounds of 32, whatever tile
//    they come from: each lane holds four i atoms and meets one queued j atom
//    per step, the pair math in packed FP32x2 instructions (eval_round); the j
//    force rotates through a group of lanes with __shfl_sync, so it returns to
//    its lane without a butterfly reduction (the reference spends 15
//    xor-shuffles per j atom).  Exclusion masks travel with the j atom; MSLD
//    pairs have a queue of their own.
//  * Accumulation in int64 fixed point (2^-32 units): i forces once per work
//    item, j forces once per queued atom, energy per pair and dU/dlambda once
//    per round.  The FP32 partial sums inside a work item have
//    a fixed order, so results do not depend on which warp, CTA or launch
//    runs which work item, nor on the order in which the items are taken.
//  * Pair math in FP32: rsqrt, erfc as exp(-x^2)*P6(1/(1+p x)) sharing the
//    Gaussian with the force (erfc_fit.h), branch-free force switching.
//  * Launched with programmatic dependent launch (launch_pdl): each kernel
//    waits for its predecessor in pdl_wait() before touching memory.
#include <cuda_runtime.h>
#include <stdint.h>

#include "bnb_internal.h"
#include "erfc_fit.h"
#include "nbdirect.h"

namespace bnb {

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;

__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ bool aabb_hit(float4 imin, float4 imax, float4 jmin, float4 jmax,
                                         float3 sh, float c2) {
  float g, acc = 0.f, lo, hi;
  lo = __fadd_rn(jmin.x, sh.x); hi = __fadd_rn(jmax.x, sh.x);
  g = fmaxf(fmaxf(__fsub_rn(lo, imax.x), __fsub_rn(imin.x, hi)), 0.f);
  acc = __fmul_rn(g, g);
  lo = __fadd_rn(jmin.y, sh.y); hi = __fadd_rn(jmax.y, sh.y);
  g = fmaxf(fmaxf(__fsub_rn(lo, imax.y), __fsub_rn(imin.y, hi)), 0.f);
  acc = __fadd_rn(acc, __fmul_rn(g, g));
  lo = __fadd_rn(jmin.z, sh.z); hi = __fadd_rn(jmax.z, sh.z);
  g = fmaxf(fmaxf(__fsub_rn(lo, imax.z), __fsub_rn(imin.z, hi)), 0.f);
  acc = __fadd_rn(acc, __fmul_rn(g, g));
  return acc <= c2;
}

// erfc(x) exp(x^2) as P6(t), t = 1/(1+p x): even/odd split halves the
// dependency chain of a plain Horner evaluation.
__device__ __forceinline__ float erfcx_poly(float t) {
  const float t2 = t * t;
  float pe = fmaf(kErfcC6, t2, kErfcC4);
  pe = fmaf(pe, t2, kErfcC2);
  pe = fmaf(pe, t2, kErfcC0);
  float po = fmaf(kErfcC5, t2, kErfcC3);
  po = fmaf(po, t2, kErfcC1);
  return fmaf(po, t, pe);
}

__device__ __forceinline__ long long to_fix(float v) {
  return __float2ll_rn(v * kFixScaleF);
}

// Sum of to_fix over a round's pairs (at most 32 a lane) without a 64-bit
// conversion per pair: v = hi 2^-12 + lo 2^-32 with both parts rounded by adding
// 1.5 2^23, whose low mantissa bits are then the integer.  hi is even in units
// of 2^-32, so the rounding of lo is the rounding of v, and the sum is that of
// to_fix bit for bit.  The four pairs of a step together, so that they share one
// test for values beyond the range (|v| >= 1000, NaN), which take to_fix itself:
// with a test per pair an energy evaluation of the 23,558-atom chain took 85.6 us,
// so 82.0 (8 MSLD replicas 243 -> 237).
struct FixSum {
  int hi = 0, lo = 0;
  __device__ __forceinline__ void add(const float2 (&v)[2], long long &sum) {
    if (!(fabsf(v[0].x) + fabsf(v[0].y) + (fabsf(v[1].x) + fabsf(v[1].y)) < 1000.f)) {
      sum += to_fix(v[0].x) + to_fix(v[0].y) + to_fix(v[1].x) + to_fix(v[1].y);
      return;
    }
    constexpr float kMagic = 12582912.f;  // 1.5 2^23
    constexpr int kMagicBits = 0x4B400000;
    const float2 magic = make_float2(kMagic, kMagic), s12 = make_float2(4096.f, 4096.f),
                 s20 = make_float2(1048576.f, 1048576.f);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const float2 th = __ffma2_rn(v[h], s12, magic);
      const float2 top = __fadd2_rn(magic, make_float2(-th.x, -th.y));
      const float2 tl = __ffma2_rn(__ffma2_rn(v[h], s12, top), s20, magic);
      hi += (__float_as_int(th.x) - kMagicBits) + (__float_as_int(th.y) - kMagicBits);
      lo += (__float_as_int(tl.x) - kMagicBits) + (__float_as_int(tl.y) - kMagicBits);
    }
  }
  __device__ __forceinline__ long long total() const { return (long long)hi * 1048576 + lo; }
};

__device__ __forceinline__ void red_add(long long *p, long long v) {
  atomicAdd(reinterpret_cast<unsigned long long *>(p), static_cast<unsigned long long>(v));
}

// ---------------------------------------------------------------------------
// Pair physics at distance r (rinv = 1/r, r2 = r*r): energy E and dE/dr.
// Electrostatics: nbdirect.cu:281-323; van der Waals: nbdirect.cu:326-396.
// Every sum says whether it is fused: left to the compiler, that differs between
// the kernels that inline this (with and without energy, MSLD, masks), and a
// replica would not have the same bits in a batch with MSLD replicas as alone.
// ---------------------------------------------------------------------------
template <int ELEC, int VDW, bool NEEDE>
__device__ __forceinline__ void pair_terms(const PairConst &pc, float r, float r2, float rinv,
                                           float qq, float c12, float c6, float &dEdr,
                                           float &E) {
  float fe, ee = 0.f;
  if (ELEC == 1) {  // PME real space
    float t = rcp_approx(fmaf(pc.pBeta, r, 1.0f));
    float p = erfcx_poly(t);
    float g = ex2_approx(pc.mBeta2Log2e * r2);
    float eel = qq * (p * g) * rinv;
    fe = -fmaf(qq * pc.twoBetaSqrtPi, g, eel) * rinv;
    ee = eel;
  } else if (ELEC == 0) {  // FSWITCH
    if (r <= pc.rswitch) {
      fe = -qq * rinv * rinv;
      if (NEEDE) ee = qq * __fadd_rn(rinv, pc.fdvc);
    } else {
      // The reference's expanded polynomial (nbdirect.cu:293-299) cancels to
      // ~0 near rCut; in FP32 that costs ~1e-5 relative force error.  The same
      // functions in factored form:
      //   dE/dr = -qq (rc^2-r^2)^2 (rc^2+2r^2-3rs^2) ginv / r^2
      //   E     =  qq (rc-r)^3 P(r) ginv / (5 r),
      //   P(r)  = 2r^3 + 6 rc r^2 + (7rc^2-5rs^2) r + 5rc^3 - 15 rc rs^2.
      float w = __fsub_rn(pc.roff2, r2);
      fe = -qq * (w * w * fmaf(2.f, r2, pc.fsC1) * pc.fsG) * (rinv * rinv);
      if (NEEDE) {
        float t = __fsub_rn(pc.rcut, r);
        float p = fmaf(fmaf(fmaf(2.f, r, pc.fsP1), r, pc.fsP2), r, pc.fsP3);
        ee = qq * (t * t * t) * p * pc.fsG5 * rinv;
      }
    }
  } else {  // FSHIFT
    float ri2 = pc.rcinv * pc.rcinv;
    fe = -qq * fmaf(rinv, rinv, -ri2);
    if (NEEDE) ee = qq * fmaf(r, ri2, fmaf(-2.f, pc.rcinv, rinv));
  }
  float rinv2 = rinv * rinv;
  float rinv3 = rinv2 * rinv;
  float rinv6 = rinv3 * rinv3;
  float el = 0.f;
  if (VDW == 0) {  // VFSWITCH, branch free
    bool in = r < pc.rswitch;
    float d3 = fmaf(rinv2, rinv, -pc.rci3), d6 = fmaf(rinv3, rinv3, -pc.rci6);
    float a = in ? rinv3 : pc.k6 * d3;
    float b = in ? rinv6 : pc.k12 * d6;
    dEdr = fmaf(fmaf(6.f * c6 * a, rinv3, -(12.f * c12 * b * rinv6)), rinv, fe);
    if (NEEDE) {
      float pe = in ? fmaf(rinv6, rinv6, -pc.dv12) : b * d6;
      float qe = in ? fmaf(rinv3, rinv3, -pc.dv6) : a * d3;
      el = fmaf(c12, pe, -(c6 * qe));
    }
  } else if (VDW == 1) {  // VSWITCH
    float f = fmaf(-12.f * c12, rinv6, 6.f * c6), e = fmaf(c12, rinv6, -c6);
    if (r < pc.rswitch) {
      dEdr = fmaf(f * rinv6, rinv, fe);
      if (NEEDE) el = e * rinv6;
    } else {
      float rijl = __fsub_rn(pc.ron2, r2), riju = __fsub_rn(pc.roff2, r2);
      float fsw = riju * riju * fmaf(-3.f, rijl, riju) * pc.rul3inv;
      float dfsw = rijl * riju * pc.rul12;
      dEdr = fmaf(fsw * f * rinv6, rinv, fmaf(dfsw * e, rinv6, fe));
      if (NEEDE) el = fsw * e * rinv6;
    }
  } else {  // VSHIFT
    float r5 = r2 * r2 * r, r6 = r2 * r2 * r2;
    float rinv12 = rinv6 * rinv6;
    dEdr = fmaf(6.f * c6, fmaf(rinv6, rinv, -(r5 * pc.vshRc12inv)),
                fmaf(-12.f * c12, fmaf(rinv12, rinv, r5 * pc.vshRc18inv), fe));
    if (NEEDE)
      el = fmaf(c12, fmaf(-3.f, pc.vshRc12inv, fmaf(2.f * r6, pc.vshRc18inv, rinv12)),
                -(c6 * fmaf(-2.f, pc.vshRc6inv, fmaf(r6, pc.vshRc12inv, rinv6))));
  }
  E = __fadd_rn(ee, el);
}

// LJ pair coefficients.  Combination mode stores per type (sqrt(12 eps),
// Rmin/2): e6 = 12 sqrt(eps_i eps_j), c6 = 2 eps Rmin^6 = e6 R6/6,
// c12 = eps Rmin^12 = e6 R6^2/12 (potential.cxx:1393-1403).
template <bool COMBINE>
__device__ __forceinline__ void lj_params(const float2 *sLJ, int rowI, int tj, float2 ljI,
                                          float2 ljJ, float &c12, float &c6) {
  if (COMBINE) {
    float e6 = ljI.x * ljJ.x;
    float R = ljI.y + ljJ.y;
    float R2 = R * R;
    float R6 = R2 * R2 * R2;
    c6 = (e6 * (1.f / 6.f)) * R6;
    c12 = (e6 * (1.f / 12.f)) * R6 * R6;
  } else {  // the shared table holds (12 c12, 6 c6)
    float2 v = sLJ[rowI + tj];
    c12 = v.x * (1.f / 12.f);
    c6 = v.y * (1.f / 6.f);
  }
}


struct KArgs {
  Dev d;
  PairConst pc;
  const float *lambda;     // [lamTotal] or null
  int count;               // count in-cutoff pairs (energy variants only)
};

// One pair at distance r = 1/rinv, r2 = r^2, of any method: returns (dE/dr)/r and
// the pair energy.  PME + VFSWITCH, the production combination, is written out
// below for two pairs at once.
template <int ELEC, int VDW, bool ENERGY, bool COMBINE>
__device__ __forceinline__ float general_pair(const PairConst &pc, float r2, float rinv, float r, float qq,
                                              const float2 *sLJ, int rowI, int tj, float2 ljI, float2 ljJ, float &E) {
  float c12, c6, dEdr;
  lj_params<COMBINE>(sLJ, rowI, tj, ljI, ljJ, c12, c6);
  pair_terms<ELEC, VDW, ENERGY>(pc, r, r2, rinv, qq, c12, c6, dEdr, E);
  return dEdr * rinv;
}

// ---------------------------------------------------------------------------
// Packed FP32x2 arithmetic (sm_100): one instruction updates the .x and .y
// halves, which the rounds below use for two independent pairs (A in .x, B in .y)
// of one lane.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 f2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 sel2(bool x, bool y, float2 a, float2 b) {
  return make_float2(x ? a.x : b.x, y ? a.y : b.y);
}

// Two PME + VFSWITCH pairs at distances r = 1/rinv, r2 = r^2 (one in .x, one in
// .y): returns (dE/dr)/r for both; with ENERGY also their energies.
//   erfc(beta r) = exp(-beta^2 r^2) P6(t),
//   VFSWITCH dE/dr * r = 6 c6 a r^-3 - 12 c12 b r^-6   (nbdirect.cu:336-346)
// with a, b = (r^-3, r^-6) inside rSwitch and (k6 (r^-3 - rc^-3),
// k12 (r^-6 - rc^-6)) outside; k6, k12 > 1 and the two forms meet at rSwitch,
// so a and b are the smaller of each.  In combination mode this is
// e6 w (a - w b) with w = Rmin^6 r^-3.  Table mode takes (12 c12, 6 c6), combine
// mode (e6, R) = (sqrt(12 eps_i) sqrt(12 eps_j), Rmin/2_i + Rmin/2_j).  nqq is
// the negative charge product and nb = -b, so no sign costs an instruction.
template <bool ENERGY, bool COMBINE, bool MSLD>
__device__ __forceinline__ float2 pme_vfsw_pair2(const PairConst &pc, float2 r2, float2 rinv,
                                                 float2 r, float2 nqq, float2 lj0, float2 lj1, float2 &E) {
  const float2 targ = fma2(f2(pc.pBeta), r, f2(1.0f));
  const float2 t = make_float2(rcp_approx(targ.x), rcp_approx(targ.y));
  const float2 garg = mul2(f2(pc.mBeta2Log2e), r2);
  const float2 g = make_float2(ex2_approx(garg.x), ex2_approx(garg.y));
  const float2 t2 = mul2(t, t);
  float2 pe = fma2(f2(kErfcC6), t2, f2(kErfcC4));
  pe = fma2(pe, t2, f2(kErfcC2));
  pe = fma2(pe, t2, f2(kErfcC0));
  float2 po = fma2(f2(kErfcC5), t2, f2(kErfcC3));
  po = fma2(po, t2, f2(kErfcC1));
  const float2 p = fma2(po, t, pe);
  const float2 nqg = mul2(nqq, g);
  const float2 rinv2 = mul2(rinv, rinv);
  const float2 rinv3 = mul2(rinv2, rinv);
  const float2 rinv6 = mul2(rinv3, rinv3);
  const float2 ao = fma2(f2(pc.k6), rinv3, f2(-pc.k6rci3));
  const float2 nbo = fma2(f2(-pc.k12), rinv6, f2(pc.k12rci6));
  const float2 a = make_float2(fminf(rinv3.x, ao.x), fminf(rinv3.y, ao.y));
  const float2 nb = make_float2(fmaxf(-rinv6.x, nbo.x), fmaxf(-rinv6.y, nbo.y));
  float2 flr, c12, c6;
  if (COMBINE) {  // lj0 = e6, lj1 = R
    const float2 R2 = mul2(lj1, lj1);
    const float2 R6 = mul2(mul2(R2, R2), R2);
    const float2 w = mul2(R6, rinv3);
    flr = mul2(mul2(lj0, w), fma2(w, nb, a));
    if (ENERGY) {
      c6 = mul2(mul2(lj0, f2(1.f / 6.f)), R6);
      c12 = mul2(mul2(mul2(lj0, f2(1.f / 12.f)), R6), R6);
    }
  } else {        // lj0 = 12 c12, lj1 = 6 c6
    flr = fma2(mul2(lj1, a), rinv3, mul2(mul2(lj0, nb), rinv6));
    if (ENERGY) {
      c12 = mul2(lj0, f2(1.f / 12.f));
      c6 = mul2(lj1, f2(1.f / 6.f));
    }
  }
  if (ENERGY) {
    const bool inA = r.x < pc.rswitch, inB = r.y < pc.rswitch;
    const float2 pe_in = fma2(rinv6, rinv6, f2(-pc.dv12));
    const float2 pe_out = mul2(nb, sub2(f2(pc.rci6), rinv6));
    const float2 qe_in = sub2(f2(pc.dv6), rinv6);
    const float2 qe_out = mul2(a, sub2(f2(pc.rci3), rinv3));
    const float2 pe2 = sel2(inA, inB, pe_in, pe_out);
    const float2 nqe2 = sel2(inA, inB, qe_in, qe_out);
    const float2 lj = fma2(c12, pe2, mul2(c6, nqe2));
    // the order of pair_terms for MSLD pairs, whose large terms may cancel
    if (MSLD) E = add2(mul2(mul2(mul2(nqq, f2(-1.f)), mul2(p, g)), rinv), lj);
    else E = fma2(mul2(mul2(nqg, f2(-1.f)), p), rinv, lj);
  }
  // Coulomb part of (dE/dr) r: -qq g (p / r + 2 beta / sqrt(pi))
  return mul2(fma2(nqg, fma2(p, rinv, f2(pc.twoBetaSqrtPi)), flr), rinv2);
}

// Per-lane loads of one candidate tile: the j slot of this lane.  Empty slots
// hold a position far outside every cutoff (k_pack).
template <bool COMBINE, int ALCH>
struct TileFetch {
  int jBlock, code, t, siteBlock;
  float4 xj;
  float2 lj;
  uint32_t mask;  // i lanes this j atom may meet
  __device__ __forceinline__ void fetch(const Dev &d, int4 cand, int c, int lane) {
    jBlock = __shfl_sync(kFull, cand.x, c);
    code = __shfl_sync(kFull, cand.y, c);
    const int mIdx = __shfl_sync(kFull, cand.z, c);
    const int jslot = 32 * jBlock + lane;
    xj = d.xyzq[jslot];
    if (COMBINE) lj = d.slotLj[jslot];
    else t = d.slotType[jslot];
    siteBlock = ALCH ? d.slotSiteBlock[jslot] : 0;
    mask = mIdx >= 0 ? d.masks[32 * (size_t)mIdx + lane] : kFull;
  }
};

// ---------------------------------------------------------------------------
// Rounds.  The j atoms of a work item's tiles that can reach the i block are
// queued per warp in shared memory with all that a pair needs of them (shifted
// position and charge, LJ parameters, accumulator slot, the i lanes they may
// meet), whatever tile they come from, and evaluated in rounds of up to 32.
//
// The i block is two halves of 16 atoms, lower and upper in z (its column is
// sorted by z), each with an AABB of its own, and each half has its own queue:
// a j atom that reaches one half only is not paired with the other.  The two
// queues are interleaved, place p of the lower in .x and of the upper in .y.
//
// In a round lane l = 8 g + r holds four i atoms, r and r + 8 of either half, so
// every group g of 8 lanes covers the block, and group g owns S of the 4 S
// places (S = 8, 4, 2 or 1).  At step k the lane meets place (r + k) mod S of its
// group: it reads the two entries from shared memory, meets the lower one with
// its two lower atoms and the upper one with its two upper atoms as two packed
// FP32x2 pairs, and hands the entries' force accumulators to the lane before
// it, so after S steps every accumulator is back in its lane; groups of S lanes
// of one group hold the same entries and are summed by xor shuffles, and each
// entry's force is added to the fixed-point accumulators once.
//
// Bound by the issue of FP32 and the latencies inside a step.  A step of four
// pairs issues 6 shared-memory loads, which depend on nothing and whose register
// pairs are the packed operands as they are, and 6 shuffles; rounds that
// rotated the j atom through shuffles against the whole block needed 18
// shuffles in a chain and 1.2 (rCut 12 A) to 1.3 times (9 A) the steps.
//
// An entry whose mask is not full (an excluded partner, a tile against
// itself) makes its round test the mask per pair; there are few of them.
// MSLD pairs (ALCH) have queues of their own: every j atom of an i block with
// MSLD atoms, and MSLD j atoms of other blocks.
// ---------------------------------------------------------------------------
// Places of the two queues.  A round is due when both halves have 32 entries, or
// when one half could overflow with the next tile, so the halves may differ by up
// to places - 64 entries before a round runs half empty.  The number decides which
// entries share a round, and with it the order of the FP32 sums, so it is the same
// in every kernel: a replica without MSLD atoms gives the same bits in a batch with
// MSLD replicas as alone.
// Measured: plain, 64 places are 0.5-1 % slower than 96, 128 no faster; MSLD, 96
// leave too little L1 (batch of 32 small boxes 90 us against 76).  96 instead of
// 64 plain places beside the MSLD queue cost no more than 1 % (32 MSLD boxes 55.8
// against 55.4 us a force evaluation, 8 solvated replicas 178 us either way).
constexpr int kPlainPlaces = 96, kMsldPlaces = 64;

template <bool COMBINE, bool MSLD, int PLACES>
struct Queue {
  static constexpr int kPlaces = PLACES;
  // .x lower, .y upper half's entry; x, y, z negated, so that a difference is an addition
  float2 x[PLACES], y[PLACES], z[PLACES], q[PLACES];
  float2 e[COMBINE ? PLACES : 1], R[COMBINE ? PLACES : 1];  // sqrt(12 eps), Rmin/2
  int2 t[COMBINE ? 1 : PLACES];                        // type index
  int2 slot[PLACES];
  uint2 mask[PLACES];
  int2 b[MSLD ? PLACES : 1];      // siteBlock
  float2 lam[MSLD ? PLACES : 1];  // its lambda
};

// One half's part of a place (an element of each array).
__device__ __forceinline__ float &half_of(float2 &v, bool up) { return up ? v.y : v.x; }
__device__ __forceinline__ int &half_of(int2 &v, bool up) { return up ? v.y : v.x; }
__device__ __forceinline__ uint32_t &half_of(uint2 &v, bool up) { return up ? v.y : v.x; }

// The four i atoms of a lane: [h].x atom r + 8 h, [h].y atom 16 + r + 8 h.
struct IAtoms {
  float2 x[2], y[2], z[2], nq[2];  // nq: negative scaled charge
  float2 e6[2], R[2];  // combine mode: (sqrt(12 eps), Rmin/2)
  int2 row[2];         // table mode: type * nTypes
};

// Sums over the groups of a warp a value per i atom (laid out as in IAtoms):
// lane l receives the total of atom l.
__device__ __forceinline__ float sum_groups(const float2 (&f)[2], int lane) {
  const bool up = lane & 16, odd = lane & 8;
  float k0 = up ? f[0].y : f[0].x, k1 = up ? f[1].y : f[1].x;
  k0 += __shfl_xor_sync(kFull, up ? f[0].x : f[0].y, 16);
  k1 += __shfl_xor_sync(kFull, up ? f[1].x : f[1].y, 16);
  return (odd ? k1 : k0) + __shfl_xor_sync(kFull, odd ? k0 : k1, 8);
}

// MSLD scaling of one pair (nbdirect.cu:244-254).
__device__ __forceinline__ bool same_site(int bi, int bj) { return ((bi ^ bj) & 0xFFFF0000) == 0; }
__device__ __forceinline__ float msld_scale(int bi, int bj, float li, float lj) {
  return same_site(bi, bj) ? (bi == bj ? lj : 0.f) : li * lj;
}

// KIND 0: no masks; 1: masks; 2: masks and MSLD scaling; 3: also soft core.
template <int ELEC, int VDW, bool ENERGY, bool COMBINE, int KIND, class Q>
__device__ __forceinline__ void eval_round(const Dev &d, const PairConst &pc, const float2 *sLJ, const Q &q, int head,
                                           int CL, int CU, int S, int lane, int iBlock, const IAtoms &I,
                                           const float *sLam, long long *sAccL, float2 (&fx)[2], float2 (&fy)[2],
                                           float2 (&fz)[2], long long &ei, unsigned long long &pairs, int count) {
  constexpr bool MSLD = KIND >= 2;
  const int r = lane & 7, base = head + (lane >> 3) * S;
  float2 jfx = f2(0.f), jfy = f2(0.f), jfz = f2(0.f), jfl = f2(0.f);
  FixSum sum;
  int2 bi[2];
  float2 li[2], fl[2];
  if (MSLD) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      bi[h].x = d.slotSiteBlock[32 * iBlock + r + 8 * h];
      bi[h].y = d.slotSiteBlock[32 * iBlock + 16 + r + 8 * h];
      li[h] = make_float2(bi[h].x ? sLam[bi[h].x & 0xFFFF] : 1.f, bi[h].y ? sLam[bi[h].y & 0xFFFF] : 1.f);
      fl[h] = f2(0.f);
    }
  }
  for (int k = 0; k < S; k++) {
    const int e = base + ((r + k) & (S - 1));
    const float2 xj = q.x[e], yj = q.y[e], zj = q.z[e], qj = q.q[e];
    float2 ej = f2(0.f), Rj = f2(0.f);
    int2 tj = make_int2(0, 0);
    if (COMBINE) {
      ej = q.e[e];
      Rj = q.R[e];
    } else {
      tj = q.t[e];
    }
    uint2 m = make_uint2(0, 0);
    if (KIND >= 1) {
      m = q.mask[e];
      m.x >>= r;
      m.y >>= r;
    }
    int2 bj = make_int2(0, 0);
    float2 lamj = f2(1.f), Es[2];  // Es: energies of the step's pairs
    if (MSLD) {
      bj = q.b[e];
      lamj = q.lam[e];
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const float2 dx = add2(I.x[h], xj), dy = add2(I.y[h], yj), dz = add2(I.z[h], zj);
      const float2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
      bool actA = r2.x < pc.rc2, actB = r2.y < pc.rc2;
      if (KIND >= 1) {
        actA = actA && (m.x & (1u << (8 * h)));
        actB = actB && (m.y & (1u << (8 * h)));
      }
      const float2 nqq = mul2(I.nq[h], qj);
      const float2 rinv = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
      const float2 rr = mul2(r2, rinv);
      float2 s, re = rr, re2 = r2, reinv = rinv, dredr, dredll;
      bool softA = false, softB = false;
      if (MSLD) {
        s = make_float2(msld_scale(bi[h].x, bj.x, li[h].x, lamj.x), msld_scale(bi[h].y, bj.y, li[h].y, lamj.y));
        dredr = f2(1.f);
        dredll = f2(0.f);
        if (KIND == 3) {  // soft core, nbdirect.cu:257-275
          const float2 rs = fma2(f2(-pc.softR), s, f2(pc.softR));
          auto soften = [&](float r1, float rs1, float &re1, float &re21, float &reinv1, float &dr, float &dl) {
            const float u = __fdividef(r1, rs1);
            const float f = fmaf(u * u * u, fmaf(-0.5f, u, 1.f), 0.5f);
            dr = (3.f - 2.f * u) * u * u;
            dl = -pc.softR * (f - dr * u);
            re1 = f * rs1;
            reinv1 = rcp_approx(re1);
            re21 = re1 * re1;
          };
          softA = (bi[h].x | bj.x) != 0 && rr.x < rs.x;
          softB = (bi[h].y | bj.y) != 0 && rr.y < rs.y;
          if (softA) soften(rr.x, rs.x, re.x, re2.x, reinv.x, dredr.x, dredll.x);
          if (softB) soften(rr.y, rs.y, re.y, re2.y, reinv.y, dredr.y, dredll.y);
        }
      }
      float2 fs, E = f2(0.f);
      constexpr bool needE = ENERGY || MSLD;
      if (ELEC == 1 && VDW == 0) {
        float2 lj0, lj1;
        if (COMBINE) {
          lj0 = mul2(I.e6[h], ej);
          lj1 = add2(I.R[h], Rj);
        } else {
          const float2 vA = sLJ[I.row[h].x + tj.x], vB = sLJ[I.row[h].y + tj.y];
          lj0 = make_float2(vA.x, vB.x);
          lj1 = make_float2(vA.y, vB.y);
        }
        fs = pme_vfsw_pair2<needE, COMBINE, MSLD>(pc, re2, reinv, re, nqq, lj0, lj1, E);
      } else {
        fs.x = general_pair<ELEC, VDW, needE, COMBINE>(pc, re2.x, reinv.x, re.x, -nqq.x, sLJ, I.row[h].x, tj.x,
                                                       make_float2(I.e6[h].x, I.R[h].x), make_float2(ej.x, Rj.x), E.x);
        fs.y = general_pair<ELEC, VDW, needE, COMBINE>(pc, re2.y, reinv.y, re.y, -nqq.y, sLJ, I.row[h].y, tj.y,
                                                       make_float2(I.e6[h].y, I.R[h].y), make_float2(ej.y, Rj.y), E.y);
      }
      if (MSLD) {
        // fs = (dE/dr_eff) / r_eff; U = s E(r_eff(r, s)): dU/dr / r = s fs (r_eff / r) dr_eff/dr
        const float2 de = mul2(mul2(fs, re), s);  // s dE/dr_eff
        float2 dl = KIND == 3 ? fma2(de, dredll, E) : E;  // dU/ds
        fs = mul2(fs, s);
        if (KIND == 3) fs = sel2(softA, softB, mul2(mul2(de, dredr), rinv), fs);
        E = mul2(E, s);
        dl = sel2(actA, actB, dl, f2(0.f));
        // dU/dlambda routing, nbdirect.cu:400-415 (block 0 is no variable)
        const bool sA = same_site(bi[h].x, bj.x), sB = same_site(bi[h].y, bj.y);
        fl[h].x += sA ? (bi[h].x == bj.x ? dl.x : 0.f) : lamj.x * dl.x;
        fl[h].y += sB ? (bi[h].y == bj.y ? dl.y : 0.f) : lamj.y * dl.y;
        jfl.x += sA ? 0.f : li[h].x * dl.x;
        jfl.y += sB ? 0.f : li[h].y * dl.y;
      }
      // branch-free: lanes out of range (or excluded) select zero
      fs = sel2(actA, actB, fs, f2(0.f));
      fx[h] = fma2(fs, dx, fx[h]);
      fy[h] = fma2(fs, dy, fy[h]);
      fz[h] = fma2(fs, dz, fz[h]);
      // the j atoms' forces with the sign of the i side, negated below
      jfx = fma2(fs, dx, jfx);
      jfy = fma2(fs, dy, jfy);
      jfz = fma2(fs, dz, jfz);
      if (ENERGY) {
        Es[h] = sel2(actA, actB, E, f2(0.f));
        if (count) pairs += (unsigned long long)actA + (unsigned long long)actB;
      }
    }
    if (ENERGY) sum.add(Es, ei);  // in fixed point per pair: exact sums of the FP32 pair values
    auto pass = [&](float2 &v) {
      v.x = __shfl_sync(kFull, v.x, lane + 1, S);
      v.y = __shfl_sync(kFull, v.y, lane + 1, S);
    };
    pass(jfx);
    pass(jfy);
    pass(jfz);
    if (MSLD) pass(jfl);
  }
  if (ENERGY) ei += sum.total();
  for (int o = 4; o >= S; o >>= 1) {
    auto fold = [&](float2 &v) {
      v.x += __shfl_xor_sync(kFull, v.x, o);
      v.y += __shfl_xor_sync(kFull, v.y, o);
    };
    fold(jfx);
    fold(jfy);
    fold(jfz);
    if (MSLD) fold(jfl);
  }
  const int place = base - head + r;
  if (r < S) {
    const int NS = 32 * d.maxBlocks;
    const int2 js = q.slot[base + r];
    auto deliver = [&](int j, float x, float y, float z) {
      if (x == 0.f && y == 0.f && z == 0.f) return;
      red_add(&d.accF[j], to_fix(-x));
      red_add(&d.accF[NS + j], to_fix(-y));
      red_add(&d.accF[2 * NS + j], to_fix(-z));
      if (!(isfinite(x) && isfinite(y) && isfinite(z))) atomicOr(&d.ctr->status, kStatusNonFinite);
    };
    if (place < CL) deliver(js.x, jfx.x, jfy.x, jfz.x);
    if (place < CU) deliver(js.y, jfx.y, jfy.y, jfz.y);
    if (MSLD) {
      const int2 b = q.b[base + r];
      if (place < CL && jfl.x != 0.f && b.x)
        atomicAdd(reinterpret_cast<unsigned long long *>(&sAccL[b.x & 0xFFFF]),
                  static_cast<unsigned long long>(to_fix(jfl.x)));
      if (place < CU && jfl.y != 0.f && b.y)
        atomicAdd(reinterpret_cast<unsigned long long *>(&sAccL[b.y & 0xFFFF]),
                  static_cast<unsigned long long>(to_fix(jfl.y)));
    }
  }
  if (MSLD) {  // the block's dU/dlambda of this round
    const float v = sum_groups(fl, lane);  // lane l: i atom l
    const int b = d.slotSiteBlock[32 * iBlock + lane];
    if (b && v != 0.f)
      atomicAdd(reinterpret_cast<unsigned long long *>(&sAccL[b & 0xFFFF]),
                static_cast<unsigned long long>(to_fix(v)));
  }
}

// A queue's fill: entries of the lower and upper half from place `head` on.
template <int PLACES>
struct Fill {
  int nL = 0, nU = 0, head = 0;
  __device__ __forceinline__ bool due(bool last) const {
    const int most = nL > nU ? nL : nU, least = nL < nU ? nL : nU;
    return least >= 32 || most > PLACES - 32 || (last && most > 0);
  }
  __device__ __forceinline__ int place(int n) const {
    const int p = head + n;
    return p >= PLACES ? p - PLACES : p;
  }
};

// One round of a queue (places without an entry are padded with one far
// outside every cutoff).
template <int ELEC, int VDW, bool ENERGY, bool COMBINE, int ALCHQ, class Q>
__device__ __forceinline__ void run_round(const Dev &d, const PairConst &pc, const float2 *sLJ, Q &q, Fill<Q::kPlaces> &f, int lane,
                                          int iBlock, const IAtoms &I, const float *sLam, long long *sAccL,
                                          float2 (&fx)[2], float2 (&fy)[2], float2 (&fz)[2], long long &ei,
                                          unsigned long long &pairs, int count) {
  // 32, 16, 8 or 4 places, whichever pads least: 20 left over go as 16 + 4
  const int n = f.nL > f.nU ? f.nL : f.nU;
  const int cap = n > 24 ? 32 : (n > 12 ? 16 : (n > 4 ? 8 : 4));
  const int CL = f.nL < cap ? f.nL : cap, CU = f.nU < cap ? f.nU : cap;
  const int at = f.head + lane;
  if (lane < cap) {
#pragma unroll
    for (int up = 0; up < 2; up++)
      if (lane >= (up ? CU : CL)) {
        half_of(q.x[at], up) = -1.0e18f;
        half_of(q.y[at], up) = half_of(q.z[at], up) = half_of(q.q[at], up) = 0.f;
        if constexpr (COMBINE) half_of(q.e[at], up) = half_of(q.R[at], up) = 0.f;
        else half_of(q.t[at], up) = 0;
        half_of(q.mask[at], up) = 0xFFFFu;
        if constexpr (ALCHQ != 0) {
          half_of(q.b[at], up) = 0;
          half_of(q.lam[at], up) = 1.f;
        }
      }
  }
  __syncwarp();
  bool masked = false;
  if (ALCHQ == 0) {
    if (lane < cap) {
      const uint2 m = q.mask[at];
      masked = (m.x & m.y) != 0xFFFFu;
    }
    masked = __any_sync(kFull, masked);
  }
  if (ALCHQ != 0)
    eval_round<ELEC, VDW, ENERGY, COMBINE, ALCHQ ? ALCHQ + 1 : 1>(d, pc, sLJ, q, f.head, CL, CU, cap >> 2, lane, iBlock,
                                                                  I, sLam, sAccL, fx, fy, fz, ei, pairs, count);
  else if (masked)
    eval_round<ELEC, VDW, ENERGY, COMBINE, 1>(d, pc, sLJ, q, f.head, CL, CU, cap >> 2, lane, iBlock, I, sLam, sAccL, fx,
                                              fy, fz, ei, pairs, count);
  else
    eval_round<ELEC, VDW, ENERGY, COMBINE, 0>(d, pc, sLJ, q, f.head, CL, CU, cap >> 2, lane, iBlock, I, sLam, sAccL, fx,
                                              fy, fz, ei, pairs, count);
  __syncwarp();  // the entries are read; their places may be refilled
  f.head = f.place(cap);
  f.nL -= CL;
  f.nU -= CU;
}

// Per-warp shared memory of k_pair.
template <bool COMBINE, int ALCH>
struct WarpSmem {
  Queue<COMBINE, false, kPlainPlaces> plain;
  Queue<COMBINE, true, kMsldPlaces> msld;
};
template <bool COMBINE>
struct WarpSmem<COMBINE, 0> {
  Queue<COMBINE, false, kPlainPlaces> plain;
};

// Resident warps, at 128 registers: 16 in 2 CTAs.  Most variants spill a little
// there too (79 of 108; bytes stored / loaded, PME + VFSWITCH: force only 12 / 12 in
// table and 32 / 24 in combination mode, soft core 36 to 96 / 32 to 64, with energy up to
// 120 / 88).  18 warps (3 x 6, 112 registers) and 20 (4 x 5, 96) spill more: chain
// of 23,558 atoms 697 -> 724 and 738 us a ten-step pass, 32 MSLD boxes 1025 -> 1113
// and 1163; 4 CTAs of 4 the same as 2 of 8.
constexpr int kPairWarps = 8, kPairCtas = 2;

// ---------------------------------------------------------------------------
// The pair kernel.
// ALCH: 0 none, 1 MSLD scaling, 2 MSLD scaling + soft core.
// ---------------------------------------------------------------------------
template <int ELEC, int VDW, int ALCH, bool ENERGY, bool COMBINE>
__global__ void __launch_bounds__(32 * kPairWarps, kPairCtas) k_pair(KArgs A) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char smem[];
  const Dev &d = A.d;
  const PairConst &pc = A.pc;
  const int lane = threadIdx.x & 31;
  const int nT = d.nTypes;
  using Warp = WarpSmem<COMBINE, ALCH>;
  Warp &ws = reinterpret_cast<Warp *>(smem)[threadIdx.x >> 5];
  float2 *sLJ = reinterpret_cast<float2 *>(smem + kPairWarps * sizeof(Warp));
  const size_t off = kPairWarps * sizeof(Warp) + (COMBINE ? 0 : (sizeof(float2) * nT * nT + 15) & ~size_t(15));
  long long *sAccL = reinterpret_cast<long long *>(smem + off);
  float *sLam = reinterpret_cast<float *>(smem + off + (ALCH ? sizeof(long long) * d.lamTotal : 0));

  if (!COMBINE)  // (12 c12, 6 c6): the factors of the force expressions folded in
    for (int i = threadIdx.x; i < nT * nT; i += blockDim.x) {
      const float2 v = d.ljTable[i];
      sLJ[i] = make_float2(12.f * v.x, 6.f * v.y);
    }
  if (ALCH)
    for (int i = threadIdx.x; i < d.lamTotal; i += blockDim.x) {
      sAccL[i] = 0;
      sLam[i] = A.lambda[i];
    }
  __syncthreads();

  const int status = d.ctr->status;
  const int nFull = d.ctr->work[0];  // full-size items; the tail items follow
  const int nWork = (status & kStatusListInvalid) ? 0 : nFull + d.ctr->work[1];
  const int NS = 32 * d.maxBlocks;
  unsigned long long pairs = 0;

  // after the first launch of a list the items are taken longest first, in
  // the order their measured cycles gave (launch_order)
  const bool ordered = d.ctr->orderValid != 0;
  int w = 0;  // position in this launch's sequence of items
  if (lane == 0) w = atomicAdd(&d.ctr->workNext, 1);
  w = __shfl_sync(kFull, w, 0);
  while (w < nWork) {
    const int item = ordered ? d.order[w] : w;
    const long long tItem = clock64();
    const int2 wk = d.work[item < nFull ? item : d.capWork + item - nFull];
    const int iBlock = work_block(wk.x);
    const int c0 = wk.y, c1 = c0 + work_tiles(wk.x);
    const RepInfo &ri = d.rep[d.blockRep[iBlock]];
    const float4 *shifts = ri.shift;  // image shift vectors by shift code
    const float4 imin = d.bmin[iBlock], imax = d.bmax[iBlock];
    float4 hmin[2], hmax[2];  // the halves' boxes
#pragma unroll
    for (int u = 0; u < 2; u++) {
      hmin[u] = d.hmin[2 * iBlock + u];
      hmax[u] = d.hmax[2 * iBlock + u];
    }

    // per-step recull of this work item's candidates (recull.cu:41-122)
    int4 cand = make_int4(0, 0, -1, 0);
    bool hit = false;
    if (c0 + lane < c1) {
      cand = d.cand[c0 + lane];
      const float4 sv = shifts[cand.y];
      const float3 sh = make_float3(sv.x, sv.y, sv.z);
      hit = aabb_hit(imin, imax, d.bmin[cand.x], d.bmax[cand.x], sh, pc.rc2);
    }
    unsigned act = __ballot_sync(kFull, hit);

    IAtoms I;
    bool anyI = false;  // the i block holds MSLD atoms
    {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int h = k & 1, up = k >> 1, is = 32 * iBlock + (lane & 7) + 8 * k;
        float4 xi = d.xyzq[is];
        if (xi.x > 1.0e17f) xi.x = -1.0e18f;  // empty i slot: never within rCut of any j, nor of padding
        half_of(I.x[h], up) = xi.x;
        half_of(I.y[h], up) = xi.y;
        half_of(I.z[h], up) = xi.z;
        half_of(I.nq[h], up) = -xi.w;
        if (COMBINE) {
          const float2 lj = d.slotLj[is];
          half_of(I.e6[h], up) = lj.x;
          half_of(I.R[h], up) = lj.y;
          half_of(I.row[h], up) = 0;
        } else {
          half_of(I.e6[h], up) = half_of(I.R[h], up) = 0.f;
          half_of(I.row[h], up) = d.slotType[is] * nT;
        }
      }
      if (ALCH) anyI = __any_sync(kFull, d.slotSiteBlock[32 * iBlock + lane] != 0);
    }
    float2 fx[2], fy[2], fz[2];
#pragma unroll
    for (int h = 0; h < 2; h++) fx[h] = fy[h] = fz[h] = f2(0.f);
    long long ei = 0;  // fixed-point energy of this lane's pairs
    Fill<kPlainPlaces> plain;
    Fill<kMsldPlaces> msld;

    // The loads of each tile are issued one tile ahead, so their latency
    // overlaps the rounds and the queueing of the tile before.
    TileFetch<COMBINE, ALCH> nxt;
    if (act) nxt.fetch(d, cand, __ffs(act) - 1, lane);
    while (true) {
      if (plain.due(!act)) {
        run_round<ELEC, VDW, ENERGY, COMBINE, 0>(d, pc, sLJ, ws.plain, plain, lane, iBlock, I, sLam, sAccL, fx, fy, fz,
                                                 ei, pairs, A.count);
        continue;
      }
      if constexpr (ALCH != 0) {
        if (msld.due(!act)) {
          run_round<ELEC, VDW, ENERGY, COMBINE, ALCH>(d, pc, sLJ, ws.msld, msld, lane, iBlock, I, sLam, sAccL, fx, fy,
                                                      fz, ei, pairs, A.count);
          continue;
        }
      }
      if (!act) break;
      act &= act - 1;
      const TileFetch<COMBINE, ALCH> cur = nxt;
      if (act) nxt.fetch(d, cand, __ffs(act) - 1, lane);
      const float4 sv = shifts[cur.code];
      const float4 xj = make_float4(cur.xj.x + sv.x, cur.xj.y + sv.y, cur.xj.z + sv.z, cur.xj.w);
      uint32_t mask = xj.x > 1.0e17f ? 0u : cur.mask;  // empty slots would pass the test against a box of NaN
      if (cur.jBlock == iBlock && cur.code == 0) mask &= (1u << lane) - 1u;  // each pair of the block once: i < j

      const bool toM = ALCH && (anyI || cur.siteBlock != 0);
      const unsigned before = (1u << lane) - 1u;
      // per half: j atoms that can reach it (per-atom AABB test, nbdirect.cu:211)
#pragma unroll
      for (int up = 0; up < 2; up++) {
        float g, gap2;
        g = fmaxf(fmaxf(hmin[up].x - xj.x, xj.x - hmax[up].x), 0.f);
        gap2 = g * g;
        g = fmaxf(fmaxf(hmin[up].y - xj.y, xj.y - hmax[up].y), 0.f);
        gap2 = fmaf(g, g, gap2);
        g = fmaxf(fmaxf(hmin[up].z - xj.z, xj.z - hmax[up].z), 0.f);
        gap2 = fmaf(g, g, gap2);
        const uint32_t mh = up ? mask >> 16 : mask & 0xFFFFu;
        const bool jin = gap2 < pc.rc2 && mh != 0u;
        auto put = [&](auto &q, int at) {
          half_of(q.x[at], up) = -xj.x;
          half_of(q.y[at], up) = -xj.y;
          half_of(q.z[at], up) = -xj.z;
          half_of(q.q[at], up) = xj.w;
          if constexpr (COMBINE) {
            half_of(q.e[at], up) = cur.lj.x;
            half_of(q.R[at], up) = cur.lj.y;
          } else {
            half_of(q.t[at], up) = cur.t;
          }
          half_of(q.slot[at], up) = 32 * cur.jBlock + lane;
          half_of(q.mask[at], up) = mh;
        };
        const unsigned mp = __ballot_sync(kFull, jin && !toM);
        if (jin && !toM) put(ws.plain, plain.place((up ? plain.nU : plain.nL) + __popc(mp & before)));
        (up ? plain.nU : plain.nL) += __popc(mp);
        if constexpr (ALCH != 0) {
          const unsigned mm = __ballot_sync(kFull, jin && toM);
          if (jin && toM) {
            const int at = msld.place((up ? msld.nU : msld.nL) + __popc(mm & before));
            put(ws.msld, at);
            half_of(ws.msld.b[at], up) = cur.siteBlock;
            half_of(ws.msld.lam[at], up) = cur.siteBlock ? sLam[cur.siteBlock & 0xFFFF] : 1.f;
          }
          (up ? msld.nU : msld.nL) += __popc(mm);
        }
      }
    }
    // the groups hold the same i atoms: after the sum lane l has atom l
    const float fix = sum_groups(fx, lane), fiy = sum_groups(fy, lane), fiz = sum_groups(fz, lane);
    // A NaN among the j atoms makes the sums of empty i slots NaN too, and nothing
    // clears their accumulators; lane l holds atom l's position among its four.
    const float2 xl = lane & 8 ? I.x[1] : I.x[0];
    const bool empty = (lane & 16 ? xl.y : xl.x) < -1.0e17f;
    if (!empty && (fix != 0.f || fiy != 0.f || fiz != 0.f)) {
      const int islot = 32 * iBlock + lane;
      red_add(&d.accF[islot], to_fix(fix));
      red_add(&d.accF[NS + islot], to_fix(fiy));
      red_add(&d.accF[2 * NS + islot], to_fix(fiz));
      if (!(isfinite(fix) && isfinite(fiy) && isfinite(fiz))) atomicOr(&d.ctr->status, kStatusNonFinite);
    }
    if (ENERGY) {
      long long e = ei;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(kFull, e, o);
      if (lane == 0 && e != 0) red_add(&d.accE[d.blockRep[iBlock]], e);
    }
    if (lane == 0) {
      const long long dt = clock64() - tItem;
      d.itemCost[item] = dt < 0xFFFFFFFFll ? (unsigned int)dt : 0xFFFFFFFFu;
      w = atomicAdd(&d.ctr->workNext, 1);
    }
    w = __shfl_sync(kFull, w, 0);
  }
  if (A.count) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) pairs += __shfl_xor_sync(kFull, pairs, o);
    if (lane == 0 && pairs) atomicAdd(&d.ctr->pairCount, pairs);
  }
  if (ALCH) {
    __syncthreads();
    for (int i = threadIdx.x; i < d.lamTotal; i += blockDim.x)
      if (sAccL[i]) red_add(&d.accL[i], sAccL[i]);
  }
}

// Log-scale bucket of a cycle count: 8 buckets per octave, 0..255.
__device__ __forceinline__ int cost_bucket(unsigned int c) {
  c = c ? c : 1u;
  const int e = 31 - __clz(c);
  const int m = e >= 3 ? (int)(c >> (e - 3)) & 7 : (int)(c << (3 - e)) & 7;
  return 8 * e + m;
}

// Work items by decreasing measured cost, one CTA: a histogram of the costs
// in log-scale buckets, bucket offsets from the most expensive bucket down
// (a warp scan over 256 buckets), then every item placed in its bucket.
// Inside a bucket the order follows the shared-memory atomics; the results
// of the pair kernel do not depend on the order of its items.
__global__ void __launch_bounds__(1024) k_order(Dev d) {
  pdl_wait();
  __shared__ int hist[256];
  const int n = (d.ctr->status & kStatusListInvalid) ? 0 : d.ctr->work[0] + d.ctr->work[1];
  for (int b = threadIdx.x; b < 256; b += blockDim.x) hist[b] = 0;
  __syncthreads();
  // eight costs in flight per thread: the loads' latency is all it spends
  constexpr int kBatch = 8;
  for (int i0 = threadIdx.x; i0 < n; i0 += kBatch * blockDim.x) {
    unsigned int c[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; k++) c[k] = i0 + k * blockDim.x < n ? d.itemCost[i0 + k * blockDim.x] : 0u;
#pragma unroll
    for (int k = 0; k < kBatch; k++)
      if (i0 + k * blockDim.x < n) atomicAdd(&hist[cost_bucket(c[k])], 1);
  }
  __syncthreads();
  if (threadIdx.x < 32) {  // lane l owns buckets 255 - 8l .. 248 - 8l (descending)
    const int l = threadIdx.x;
    int c[8], sum = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      c[k] = hist[255 - 8 * l - k];
      sum += c[k];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(kFull, incl, o);
      if (l >= o) incl += v;
    }
    int run = incl - sum;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      hist[255 - 8 * l - k] = run;
      run += c[k];
    }
  }
  __syncthreads();
  for (int i0 = threadIdx.x; i0 < n; i0 += kBatch * blockDim.x) {
    unsigned int c[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; k++) c[k] = i0 + k * blockDim.x < n ? d.itemCost[i0 + k * blockDim.x] : 0u;
#pragma unroll
    for (int k = 0; k < kBatch; k++)
      if (i0 + k * blockDim.x < n) d.order[atomicAdd(&hist[cost_bucket(c[k])], 1)] = i0 + k * blockDim.x;
  }
  if (threadIdx.x == 0) d.ctr->orderValid = n > 0;
}

// Converts the fixed-point accumulators to the caller's outputs and clears them.
// One thread per atom, in atom order: the outputs (in the caller's atom
// order) are written coalesced, and the per-slot accumulators, still in L2
// from the pair kernel's atomics, are gathered through atomSlot.
__global__ void k_finalize(Dev d, bnb_outputs o, int mode) {
  pdl_wait();
  const int S = 32 * d.maxBlocks;
  const double inv = 1.0 / kFixScale;
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < d.N; a += gridDim.x * blockDim.x) {
    const int t = d.atomSlot[a];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const long long v = d.accF[k * S + t];
      if (v) d.accF[k * S + t] = 0;
      const double f = (double)v * inv;
      if (o.force64) out64(&o.force64[3 * a + k], f, mode);
      if (o.force) out32(&o.force[3 * a + k], (float)f, mode);
    }
  }
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) d.ctr->workNext = 0;  // the pair kernel of the next step starts at item 0
    for (int i = threadIdx.x; i < d.lamTotal; i += blockDim.x) {
      long long v = d.accL[i];
      d.accL[i] = 0;
      double f = (double)v * inv;
      if (o.lambdaForce64) out64(&o.lambdaForce64[i], f, mode);
      if (o.lambdaForce) out32(&o.lambdaForce[i], (float)f, mode);
    }
    for (int r = threadIdx.x; r < d.R; r += blockDim.x) {
      long long v = d.accE[r];
      d.accE[r] = 0;
      double e = (double)v * inv;
      if (o.energy64) out64(&o.energy64[r], e, mode);
      if (o.energy) outE(&o.energy[r], e, mode);
    }
  }
}

// Persistent launch: as many CTAs as fit at once; warps pull work items from
// the device counter, so the grid never leaves a partial last wave.  `resident`
// is the handle's own (CTAs an SM holds of this kernel at its size, 0 until
// asked for).  The shared-memory limit belongs to the kernel, which all handles
// and threads share: it is set to the most that any handle may ask for, so no
// call takes another's setting back.
template <int ELEC, int VDW, int ALCH, bool ENERGY, bool COMBINE>
void launch_t(const KArgs &a, int maxGrid, int sms, int &resident, size_t shmem, cudaStream_t s) {
  auto k = k_pair<ELEC, VDW, ALCH, ENERGY, COMBINE>;
  constexpr size_t queues = kPairWarps * sizeof(WarpSmem<COMBINE, ALCH>);
  constexpr size_t most = queues + (COMBINE ? 0 : sizeof(float2) * kMaxTableTypes * kMaxTableTypes) +
                          (ALCH ? (sizeof(long long) + sizeof(float)) * kMaxLambdaShared : 0);
  static_assert(most <= 227 * 1024, "fits an SM");
  shmem += queues;
  if (resident == 0) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, k, 32 * kPairWarps, shmem) != cudaSuccess ||
        resident < 1)
      resident = 1;
  }
  int grid = resident * sms;
  if (grid > maxGrid) grid = maxGrid;
  if (grid < 1) grid = 1;
  launch_pdl(k, grid, 32 * kPairWarps, shmem, s, a);
}

template <int ELEC, int VDW>
void launch_ev(const KArgs &a, int alch, bool energy, bool combine, int grid, int sms, int &resident, size_t shmem,
               cudaStream_t s) {
#define BNB_L(AL, EN, CO) \
  if (alch == AL && energy == EN && combine == CO) { launch_t<ELEC, VDW, AL, EN, CO>(a, grid, sms, resident, shmem, s); return; }
  BNB_L(0, false, false) BNB_L(0, false, true) BNB_L(0, true, false) BNB_L(0, true, true)
  BNB_L(1, false, false) BNB_L(1, false, true) BNB_L(1, true, false) BNB_L(1, true, true)
  BNB_L(2, false, false) BNB_L(2, false, true) BNB_L(2, true, false) BNB_L(2, true, true)
#undef BNB_L
}

// ---------------------------------------------------------------------------
// All-pairs variant for one small periodic system (bnb_nbdirect_noalloc): no
// block list; every 32x32 tile of atom blocks (J >= I) is visited by one warp
// with minimum-image distances.  Lane l keeps atom 32I+l; the j data and the
// j-force accumulators rotate one lane per step, so after 32 steps every lane
// holds its own j atom again and adds its total once.  The pair physics is
// pair_terms (the general path of the list kernel), with table LJ
// coefficients read from global memory.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool excluded_sorted(const int *ex, int lo, int hi, int j) {
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    const int v = ex[mid];
    if (v == j) return true;
    if (v < j) lo = mid + 1;
    else hi = mid;
  }
  return false;
}

template <int ELEC, int VDW, bool ENERGY>
__global__ void __launch_bounds__(128) k_allpairs(AllPairsArgs a) {
  const int lane = threadIdx.x & 31;
  const int I = blockIdx.y;
  const int J = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int nb = (a.N + 31) >> 5;
  if (J < I || J >= nb) return;  // uniform per warp
  const PairConst &pc = a.pc;
  const int i = 32 * I + lane;
  const bool iv = i < a.N;
  float xi = 0.f, yi = 0.f, zi = 0.f, qi = 0.f;
  int ti = 0, e0 = 0, e1 = 0;
  if (iv) {
    xi = a.x[3 * i]; yi = a.x[3 * i + 1]; zi = a.x[3 * i + 2];
    const bnb_nbond n = a.nb[i];
    qi = n.q * a.sqrtK;
    ti = n.typeIdx;
    e0 = a.exclStart[i];
    e1 = a.exclStart[i + 1];
  }
  const int j0 = 32 * J + lane;
  float xj = 0.f, yj = 0.f, zj = 0.f, qj = 0.f;
  int tj = 0;
  if (j0 < a.N) {
    xj = a.x[3 * j0]; yj = a.x[3 * j0 + 1]; zj = a.x[3 * j0 + 2];
    const bnb_nbond n = a.nb[j0];
    qj = n.q * a.sqrtK;
    tj = n.typeIdx;
  }
  float fix = 0.f, fiy = 0.f, fiz = 0.f, fjx = 0.f, fjy = 0.f, fjz = 0.f;
  long long ef = 0;  // energy in fixed point per pair
  const int src = (lane + 1) & 31;
  for (int k = 0; k < 32; ++k) {
    const int jl = (lane + k) & 31;
    const int j = 32 * J + jl;
    if (iv && j < a.N && (J != I || jl > lane)) {
      float dx = xi - xj, dy = yi - yj, dz = zi - zj;
      dx -= a.box.x * rintf(dx * a.boxInv.x);
      dy -= a.box.y * rintf(dy * a.boxInv.y);
      dz -= a.box.z * rintf(dz * a.boxInv.z);
      const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      if (r2 < pc.rc2 && !excluded_sorted(a.exclAtom, e0, e1, j)) {
        const float rinv = rsqrt_approx(r2);
        const float r = r2 * rinv;
        const bnb_vdw v = a.vdw[ti * a.nTypes + tj];
        float dEdr = 0.f, E = 0.f;
        pair_terms<ELEC, VDW, ENERGY>(pc, r, r2, rinv, qi * qj, v.c12, v.c6, dEdr, E);
        const float sc = dEdr * rinv;
        fix = fmaf(sc, dx, fix); fiy = fmaf(sc, dy, fiy); fiz = fmaf(sc, dz, fiz);
        fjx = fmaf(-sc, dx, fjx); fjy = fmaf(-sc, dy, fjy); fjz = fmaf(-sc, dz, fjz);
        if (ENERGY) ef += to_fix(E);
      }
    }
    xj = __shfl_sync(0xFFFFFFFFu, xj, src);
    yj = __shfl_sync(0xFFFFFFFFu, yj, src);
    zj = __shfl_sync(0xFFFFFFFFu, zj, src);
    qj = __shfl_sync(0xFFFFFFFFu, qj, src);
    tj = __shfl_sync(0xFFFFFFFFu, tj, src);
    fjx = __shfl_sync(0xFFFFFFFFu, fjx, src);
    fjy = __shfl_sync(0xFFFFFFFFu, fjy, src);
    fjz = __shfl_sync(0xFFFFFFFFu, fjz, src);
  }
  const int S = a.stride;
  if (iv) {
    red_add(&a.accF[i], to_fix(fix));
    red_add(&a.accF[S + i], to_fix(fiy));
    red_add(&a.accF[2 * S + i], to_fix(fiz));
  }
  if (j0 < a.N) {
    red_add(&a.accF[j0], to_fix(fjx));
    red_add(&a.accF[S + j0], to_fix(fjy));
    red_add(&a.accF[2 * S + j0], to_fix(fjz));
  }
  if (ENERGY) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ef += __shfl_xor_sync(0xFFFFFFFFu, ef, o);
    if (lane == 0 && ef != 0) red_add(a.accE, ef);
  }
}

// Converts the all-pairs accumulators to the outputs (bnb_compute's output
// semantics) and writes every entry it read back to zero.
__global__ void k_allpairs_finalize(AllPairsArgs a, bnb_outputs o) {
  const double inv = 1.0 / kFixScale;
  const int S = a.stride;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < a.N; t += gridDim.x * blockDim.x) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const long long v = a.accF[k * S + t];
      a.accF[k * S + t] = 0;
      const double f = (double)v * inv;
      if (o.force64) o.force64[3 * t + k] = f;
      if (o.force && v) o.force[3 * t + k] += (float)f;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const long long v = *a.accE;
    *a.accE = 0;
    const double en = (double)v * inv;
    if (o.energy64) *o.energy64 = en;
    if (o.energy) *o.energy += en;
  }
}

template <int ELEC, int VDW>
void launch_allpairs_ev(const AllPairsArgs &a, bool energy, dim3 grid, cudaStream_t s) {
  if (energy) k_allpairs<ELEC, VDW, true><<<grid, 128, 0, s>>>(a);
  else k_allpairs<ELEC, VDW, false><<<grid, 128, 0, s>>>(a);
}

}  // namespace

int launch_pair(const Dev &d, const PairConst &pc, const float *lambda, int elec, int vdw,
                int alch, bool energy, bool count, int grid, int sms, int &resident, cudaStream_t s) {
  KArgs a{d, pc, lambda, count ? 1 : 0};
  size_t shmem = d.ljCombine ? 0 : sizeof(float2) * d.nTypes * d.nTypes;
  shmem = (shmem + 15) & ~size_t(15);
  if (alch) shmem += (sizeof(long long) + sizeof(float)) * d.lamTotal;
  bool combine = d.ljCombine != 0;
  switch (elec * 3 + vdw) {
    case 0: launch_ev<0, 0>(a, alch, energy, combine, grid, sms, resident, shmem, s); break;
    case 1: launch_ev<0, 1>(a, alch, energy, combine, grid, sms, resident, shmem, s); break;
    case 2: launch_ev<0, 2>(a, alch, energy, combine, grid, sms, resident, shmem, s); break;
    case 3: launch_ev<1, 0>(a, alch, energy, combine, grid, sms, resident, shmem, s); break;
    case 4: launch_ev<1, 1>(a, alch, energy, combine, grid, sms, resident, shmem, s); break;
    case 5: launch_ev<1, 2>(a, alch, energy, combine, grid, sms, resident, shmem, s); break;
    case 6: launch_ev<2, 0>(a, alch, energy, combine, grid, sms, resident, shmem, s); break;
    case 7: launch_ev<2, 1>(a, alch, energy, combine, grid, sms, resident, shmem, s); break;
    case 8: launch_ev<2, 2>(a, alch, energy, combine, grid, sms, resident, shmem, s); break;
    default: return BNB_ERR_ARG;
  }
  return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_CUDA;
}

void launch_finalize(const Dev &d, const bnb_outputs &o, int mode, cudaStream_t s) {
  int n = d.N;
  int grid = (n + 255) / 256;
  if (grid > 148 * 8) grid = 148 * 8;
  if (grid < 1) grid = 1;
  launch_pdl(k_finalize, grid, 256, 0, s, d, o, mode);
}

void launch_order(const Dev &d, cudaStream_t s) { launch_pdl(k_order, 1, 1024, 0, s, d); }

int launch_allpairs(const AllPairsArgs &a, const bnb_outputs &o, int elec, int vdw, bool energy,
                    cudaStream_t s) {
  const int nb = (a.N + 31) / 32;
  const dim3 grid((nb + 3) / 4, nb);
  if (nb > 0) switch (elec * 3 + vdw) {
    case 0: launch_allpairs_ev<0, 0>(a, energy, grid, s); break;
    case 1: launch_allpairs_ev<0, 1>(a, energy, grid, s); break;
    case 2: launch_allpairs_ev<0, 2>(a, energy, grid, s); break;
    case 3: launch_allpairs_ev<1, 0>(a, energy, grid, s); break;
    case 4: launch_allpairs_ev<1, 1>(a, energy, grid, s); break;
    case 5: launch_allpairs_ev<1, 2>(a, energy, grid, s); break;
    case 6: launch_allpairs_ev<2, 0>(a, energy, grid, s); break;
    case 7: launch_allpairs_ev<2, 1>(a, energy, grid, s); break;
    case 8: launch_allpairs_ev<2, 2>(a, energy, grid, s); break;
    default: return BNB_ERR_ARG;
  }
  if (cudaGetLastError() != cudaSuccess) return BNB_ERR_CUDA;
  k_allpairs_finalize<<<a.N > 0 ? (a.N + 255) / 256 : 1, 256, 0, s>>>(a, o);
  return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_CUDA;
}

}  // namespace bnb
