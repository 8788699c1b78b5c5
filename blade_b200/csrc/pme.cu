// PME reciprocal space and Ewald self term (sm_100a).
//
// Counterpart of getforce_ewald and getforce_ewaldself
// (src/nbrecip/nbrecip.cu:19-555).  The algorithm is the reference's smooth
// PME: lambda-scaled charges are spread with order-n cardinal B-splines
// (grid point (floor(u) + t) mod K takes M_n(u - floor(u) + n - 1 - t),
// u = x K / L; nbrecip.cu:85-213), the unnormalised R2C spectrum is
// multiplied by B(m) exp(-pi^2 k^2 / beta^2) / (2 pi V k^2) (nbrecip.cu:
// 215-256), the C2R result is the potential grid and the gather returns
// dU/dx = 2 lambda q (K / L) sum dM M M phi, dU/dlambda = 2 q phi and
// E = lambda q phi (nbrecip.cu:258-465).  Charges arrive scaled by
// sqrt(kElectric), so the influence function carries no kElectric.
// Differences by design:
//   * the charge grid accumulates in int64 fixed point (2^-32), so the grid,
//     and with it every output, is identical run to run;
//   * u is formed in FP64 and wrapped, so any unwrapped coordinate lands on
//     the right grid point;
//   * lanes own z offsets (contiguous grid addresses within one instruction)
//     instead of x/y/z parity classes, and the atoms of a molecule are spread
//     together;
//   * R replicas with their own grids in one launch per phase.
// Triclinic cells (the reference's flagBox branch): the fractional
// coordinates s = H^-1 x of the cell matrix H (columns A, B, C) replace x / L
// (nbrecip.cu:116-178), here by back substitution in FP64; the wave vectors
// are H^-T m (nbrecip.cu:236-242) and dU/dx = H^-T dU/ds (nbrecip.cu:456-462),
// with H^-1 as the reference's State::kTricBox_f (state.cxx:485-491).
// Orthorhombic handles keep the plain per-dimension path.
// The 3-D transforms are pmefft.cu's, for all replicas at once.  Grids outside
// its range (a plane above 220 KB of shared memory, about 165^2, or an edge with
// a prime factor above 5) are cuFFT plans, one batched plan per set of equal
// grids, as in the reference.
#include <cuda_runtime.h>

#include "pme.h"

namespace bnb {
namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr double kPi = 3.14159265358979323846;

__device__ __forceinline__ long long to_fix(float v) { return __float2ll_rn(v * kFixScaleF); }

__device__ __forceinline__ void red_add(long long *p, long long v) {
  atomicAdd(reinterpret_cast<unsigned long long *>(p), static_cast<unsigned long long>(v));
}

// w[t] = M_n(f + n - 1 - t) and dw[t] = M_n'(f + n - 1 - t), t = 0..n-1, from
// the Cox-de Boor recursion M_k(x) = (x M_{k-1}(x) + (k - x) M_{k-1}(x - 1))
// / (k - 1) on the points x = f + j, and M_n'(x) = M_{n-1}(x) - M_{n-1}(x-1).
template <int ORDER>
__device__ __forceinline__ void bspline(float f, float (&w)[ORDER], float (&dw)[ORDER]) {
  float a[ORDER];
  float prev[ORDER];
  a[0] = 1.f;
#pragma unroll
  for (int j = 1; j < ORDER; j++) a[j] = 0.f;
#pragma unroll
  for (int k = 2; k <= ORDER; k++) {
    if (k == ORDER) {
#pragma unroll
      for (int j = 0; j < ORDER; j++) prev[j] = a[j];
    }
    const float inv = 1.f / (float)(k - 1);
#pragma unroll
    for (int j = k - 1; j >= 0; j--) {
      const float x = f + (float)j;
      const float left = j < k - 1 ? a[j] : 0.f;
      const float right = j >= 1 ? a[j - 1] : 0.f;
      a[j] = fmaf(x, left, ((float)k - x) * right) * inv;
    }
  }
#pragma unroll
  for (int t = 0; t < ORDER; t++) {
    const int j = ORDER - 1 - t;
    w[t] = a[j];
    dw[t] = (j < ORDER - 1 ? prev[j] : 0.f) - (j >= 1 ? prev[j - 1] : 0.f);
  }
}

// First grid index (mod K) and fraction of an atom along dimension `dim` of its
// replica's cell.  The fractional coordinate is formed in FP64 and reduced to
// [0, 1) before it is scaled, so any unwrapped coordinate lands on its grid point.
__device__ __forceinline__ void grid_coord(const PmeArgs &a, const float *x, int K, const RepInfo &ri, int dim,
                                           int &i0, float &frac) {
  double f;
  if (!a.tric) {
    f = (double)x[dim] * ri.inv[dim];
  } else {  // box = (A_x, B_y, C_z), tric = (B_x, C_x, C_y)
    const double sz = (double)x[2] * ri.inv[2];
    const double sy = ((double)x[1] - (double)ri.tric[2] * sz) * ri.inv[1];
    f = dim == 2 ? sz : (dim == 1 ? sy : ((double)x[0] - (double)ri.tric[0] * sy - (double)ri.tric[1] * sz) * ri.inv[0]);
  }
  const double u = (f - floor(f)) * (double)K, u0 = floor(u);
  frac = (float)(u - u0);
  i0 = (int)u0;
  if ((unsigned)i0 >= (unsigned)K) i0 = 0;  // f rounds to 1 (a tiny negative number), or is no number
}

__device__ __forceinline__ float atom_scale(const PmeArgs &a, int atom, int &block) {
  block = a.siteBlock[atom] & 0xFFFF;
  return (block && a.lambda) ? a.lambda[block] : 1.f;
}

// ---------------------------------------------------------------------------
// Spread.  A warp takes 9 consecutive atoms: lanes 3 j + dim evaluate their
// splines (one coordinate and one spline per warp instead of three per atom)
// into shared memory; then runs of up to 4 neighbouring atoms whose first grid
// points lie within (8 - ORDER) / 2 of the run's first atom's (the atoms of a
// molecule) are spread together over a box of 8 points an edge, lane = 4 rows of
// y x 8 z, two rows of y per lane: the atoms' fixed-point values of a point are
// summed in registers and added to the grid once.  The values and the sums are
// those of one addition per atom.
//
// Bound by the L2's atomic additions (0.52 T/s of 64 bits) and the issue of the
// fixed-point conversions: one addition per atom and point is 216 an atom at
// order 6; a water's three atoms together touch about 330 points, not 648.
// Measured at order 6: 192,000 atoms 80 -> 50 us, 20,577 atoms 16 -> 13.6 us.
// ---------------------------------------------------------------------------
constexpr int kSpreadAtoms = 9;

// The box of one run of NA atoms, x plane by x plane.  bx, by, bz: weights of the
// box's points by atom (.x .. .w), zero outside an atom's own points; bz carries
// the charge in fixed-point units.
template <int NA>
__device__ __forceinline__ void spread_box(const float4 *bx, float4 by0, float4 by1, float4 bz, long long *base,
                                           int row0, int row1, int x0, int K0, int plane) {
  auto get = [](const float4 &v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : (k == 2 ? v.z : v.w)); };
#pragma unroll 2
  for (int x = 0; x < 8; x++) {
    const float4 w = bx[x];
    bool any = false;
#pragma unroll
    for (int k = 0; k < NA; k++) any = any || get(w, k) != 0.f;
    if (!any) continue;  // uniform
    long long s0 = 0, s1 = 0;
#pragma unroll
    for (int k = 0; k < NA; k++) {
      const float q = get(bz, k) * get(w, k);
      s0 += __float2ll_rn(q * get(by0, k));
      s1 += __float2ll_rn(q * get(by1, k));
    }
    int ix = x0 + x;
    if (ix >= K0) ix -= K0;
    if (ix >= K0) ix -= K0;  // a box may be longer than a short edge
    long long *p = base + (size_t)ix * plane;
    if (s0) red_add(p + row0, s0);
    if (s1) red_add(p + row1, s1);
  }
}

template <int ORDER, bool SMALL>
__global__ void __launch_bounds__(256) k_spread(PmeArgs a) {
  pdl_wait();
  constexpr int perWarp = SMALL ? 3 : kSpreadAtoms;
  constexpr int RANGE = (8 - ORDER) / 2;
  __shared__ float sW[8][kSpreadAtoms][3][8];
  __shared__ float4 sB[8][3][8];  // a run's box: [dim][point], component = atom
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int first = (blockIdx.x * 8 + wp) * perWarp;
  if (first >= a.N) return;  // uniform per warp
  const int cnt = a.N - first < perWarp ? a.N - first : perWarp;
  int mine = 0;  // lane 3 j + dim: first grid index of atom j along dim
  {
    const int j = lane / 3, dim = lane - 3 * j;
    if (lane < 3 * cnt) {
      const int atom = first + j, r = a.atomRep[atom];
      float frac, w[ORDER], d[ORDER];
      grid_coord(a, a.x + 3 * atom, a.prep[r].K[dim], a.rep[r], dim, mine, frac);
      bspline<ORDER>(frac, w, d);
#pragma unroll
      for (int k = 0; k < ORDER; k++) sW[wp][j][dim][k] = w[k];
    }
  }
  // lane j: atom j's first grid indices, charge and replica
  int g[3], rep = -1;
#pragma unroll
  for (int k = 0; k < 3; k++) g[k] = __shfl_sync(kFull, mine, 3 * lane + k);
  float q = 0.f;
  if (lane < cnt) {
    int block;
    q = a.q[first + lane] * atom_scale(a, first + lane, block);
    rep = a.atomRep[first + lane];
  }
  __syncwarp();
  const int z = lane & 7, y = lane >> 3;
  unsigned left = __ballot_sync(kFull, q != 0.f);
  while (left) {
    const int h = __ffs(left) - 1;
    const int r = __shfl_sync(kFull, rep, h);
    const PmeRep &pr = a.prep[r];
    const int K0 = pr.K[0], K1 = pr.K[1], K2 = pr.K[2];
    // offsets from the run's first atom; the run ends at the first that is not near
    int c[3], e[3];
    bool near = rep == r;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const int K = pr.K[k];
      c[k] = __shfl_sync(kFull, g[k], h);
      e[k] = g[k] - c[k];
      e[k] = 2 * e[k] > K ? e[k] - K : (2 * e[k] < -K ? e[k] + K : e[k]);
      near = near && e[k] >= -RANGE && e[k] <= RANGE;
    }
    const unsigned run = __ballot_sync(kFull, near) >> h;
    const int len = __ffs(~run) - 1, n = len < 4 ? len : 4;
    {  // lane 8 k + i: the weights of atom h + k at point i of the box
      const int k = lane >> 3, i = lane & 7, at = (h + k) & 31;
      const int e0 = __shfl_sync(kFull, e[0], at), e1 = __shfl_sync(kFull, e[1], at), e2 = __shfl_sync(kFull, e[2], at);
      const float qk = __shfl_sync(kFull, q, at) * kFixScaleF;  // a power of two: exact
      float w0 = 0.f, w1 = 0.f, w2 = 0.f;
      if (k < n) {
        const float(&w)[3][8] = sW[wp][h + k];
        const int t0 = i - RANGE - e0, t1 = i - RANGE - e1, t2 = i - RANGE - e2;
        if ((unsigned)t0 < (unsigned)ORDER) w0 = w[0][t0];
        if ((unsigned)t1 < (unsigned)ORDER) w1 = w[1][t1];
        if ((unsigned)t2 < (unsigned)ORDER) w2 = qk * w[2][t2];
      }
      __syncwarp();  // the run before has been read
      reinterpret_cast<float *>(&sB[wp][0][i])[k] = w0;
      reinterpret_cast<float *>(&sB[wp][1][i])[k] = w1;
      reinterpret_cast<float *>(&sB[wp][2][i])[k] = w2;
      __syncwarp();
    }
    // grid index of a box point; a box may be longer than a short edge
    auto wrapped = [](int i, int K) {
      if (i < 0) i += K;
      if (i >= K) i -= K;
      if (i >= K) i -= K;
      return i;
    };
    int x0 = c[0] - RANGE;
    if (x0 < 0) x0 += K0;
    long long *base = a.qfix + pr.gridOff + wrapped(c[2] - RANGE + z, K2);
    const int row0 = wrapped(c[1] - RANGE + y, K1) * K2, row1 = wrapped(c[1] - RANGE + y + 4, K1) * K2;
    const float4 by0 = sB[wp][1][y], by1 = sB[wp][1][y + 4], bz = sB[wp][2][z];
    switch (n) {
      case 1: spread_box<1>(sB[wp][0], by0, by1, bz, base, row0, row1, x0, K0, K1 * K2); break;
      case 2: spread_box<2>(sB[wp][0], by0, by1, bz, base, row0, row1, x0, K0, K1 * K2); break;
      case 3: spread_box<3>(sB[wp][0], by0, by1, bz, base, row0, row1, x0, K0, K1 * K2); break;
      default: spread_box<4>(sB[wp][0], by0, by1, bz, base, row0, row1, x0, K0, K1 * K2); break;
    }
    left &= ~(((1u << n) - 1u) << h);
  }
}

// Fixed point -> FP32 grid, clearing the fixed-point grid for the next call.
__global__ void k_fix_to_grid(PmeArgs a) {
  pdl_wait();
  const double inv = 1.0 / kFixScale;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.totalGrid; i += gridDim.x * blockDim.x) {
    const long long v = a.qfix[i];
    a.grid[i] = (float)((double)v * inv);
    if (v) a.qfix[i] = 0;
  }
}

// ---------------------------------------------------------------------------
// Convolution between cuFFT transforms: blockIdx.y = replica, threads stride
// over its half spectrum.
// ---------------------------------------------------------------------------
__global__ void k_convolve(PmeArgs a) {
  pdl_wait();
  const int r = blockIdx.y;
  const PmeRep pr = a.prep[r];
  const RepInfo &ri = a.rep[r];
  const int K1 = pr.K[1], K2h = pr.K[2] / 2 + 1, n = pr.K[0] * K1 * K2h;
  const InfluenceFn fn(a, pr, ri);
  float2 *spec = a.cplx + pr.cplxOff;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const int k = e % K2h;
    const int row = e / K2h;
    const int j = row % K1;
    const int i = row / K1;
    const float factor = fn(i, j, k);
    float2 v = spec[e];
    v.x *= factor;
    v.y *= factor;
    spec[e] = v;
  }
}

// lambda and energy accumulators -> outputs, by the calling CTA's threads.
__device__ void finalize_outputs(const PmeArgs &a, const bnb_outputs &o, bool energy) {
  const double inv = 1.0 / kFixScale;
  for (int i = threadIdx.x; i < a.lamTotal; i += blockDim.x) {
    const long long v = __ldcg(&a.accL[i]);
    a.accL[i] = 0;
    const double f = (double)v * inv;
    if (o.lambdaForce64) out64(&o.lambdaForce64[i], f, a.mode);
    if (o.lambdaForce) out32(&o.lambdaForce[i], (float)f, a.mode);
  }
  if (energy)
    for (int r = threadIdx.x; r < a.R; r += blockDim.x) {
      const long long v = __ldcg(&a.accE[r]);
      a.accE[r] = 0;
      const double e = (double)v * inv;
      if (o.energy64) out64(&o.energy64[r], e, a.mode);
      if (o.energy) outE(&o.energy[r], e, a.mode);
    }
}

// The last CTA of a launch to finish writes the lambda and energy outputs
// (every CTA's reductions are fenced before it takes its ticket), so no
// separate finalize launch follows the gather.
__device__ void finalize_if_last(const PmeArgs &a, const bnb_outputs &o, bool energy) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(a.done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  finalize_outputs(a, o, energy);
  if (threadIdx.x == 0) *a.done = 0;  // ready for the next launch
}

// ---------------------------------------------------------------------------
// Gather.  A warp takes 8 atoms: lanes 3 j + dim evaluate their splines into
// shared memory, then 8 lanes per atom gather, 4 atoms at a time: lane g owns z
// offset g and visits the ORDER x ORDER (x, y) offsets; the 8 lanes of an atom
// reduce with xor shuffles and lanes 0-2 write its force.
//
// Bound by the latency of its loads, so by the warps in flight: 64 registers (4
// CTAs per SM) 138 us an evaluation of 192,000 atoms, 80 registers 151, 48 with
// spills 162.  Gathering a molecule's atoms together, as the spread does, loads
// half as much and was slower (150 us): it is not the loads' number that bounds.
// ---------------------------------------------------------------------------
constexpr int kGatherAtoms = 8;
template <int ORDER, bool ENERGY, bool SMALL>
__global__ void __launch_bounds__(256, 4) k_gather(PmeArgs a, bnb_outputs o) {
  pdl_wait();
  constexpr int perWarp = SMALL ? 4 : kGatherAtoms;
  __shared__ float sW[8][kGatherAtoms][3][8], sD[8][kGatherAtoms][3][8];
  __shared__ int sI[8][kGatherAtoms][4];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, g = lane & 7;
  const int first = (blockIdx.x * 8 + wp) * perWarp;
  {
    const int j = lane / 3, dim = lane - 3 * j, atom = first + j;
    if (lane < 3 * perWarp && atom < a.N) {
      const int r = a.atomRep[atom];
      int i0;
      float frac, w[ORDER], d[ORDER];
      grid_coord(a, a.x + 3 * atom, a.prep[r].K[dim], a.rep[r], dim, i0, frac);
      bspline<ORDER>(frac, w, d);
#pragma unroll
      for (int k = 0; k < ORDER; k++) {
        sW[wp][j][dim][k] = w[k];
        sD[wp][j][dim][k] = d[k];
      }
      sI[wp][j][dim] = i0;
      if (dim == 0) sI[wp][j][3] = r;
    }
  }
  __syncwarp();
#pragma unroll 1
  for (int half = 0; half < perWarp / 4; half++) {
    const int j = 4 * half + (lane >> 3), atom = first + j;
    const bool valid = atom < a.N;
    float phi = 0.f, gx = 0.f, gy = 0.f, gz = 0.f, qe = 0.f, qraw = 0.f;
    int r = 0, block = 0;
    PmeRep pr{};
    if (valid) {
      r = sI[wp][j][3];
      pr = a.prep[r];
      qraw = a.q[atom];
      qe = qraw * atom_scale(a, atom, block);
    }
    if (valid && g < ORDER) {
      const int K0 = pr.K[0], K1 = pr.K[1], K2 = pr.K[2];
      int iz = sI[wp][j][2] + g;
      if (iz >= K2) iz -= K2;
      const float *base = a.grid + pr.gridOff + iz;
      int oy[ORDER];
      float wy[ORDER], dy[ORDER];
#pragma unroll
      for (int ty = 0; ty < ORDER; ty++) {
        int iy = sI[wp][j][1] + ty;
        if (iy >= K1) iy -= K1;
        oy[ty] = iy * K2;
        wy[ty] = sW[wp][j][1][ty];
        dy[ty] = sD[wp][j][1][ty];
      }
#pragma unroll
      for (int tx = 0; tx < ORDER; tx++) {
        int ix = sI[wp][j][0] + tx;
        if (ix >= K0) ix -= K0;
        const float *plane = base + (size_t)ix * (K1 * K2);
        const float wx = sW[wp][j][0][tx], dx = sD[wp][j][0][tx];
        float p = 0.f, py = 0.f;  // sum over y of P wy, P dy
#pragma unroll
        for (int ty = 0; ty < ORDER; ty++) {
          const float P = __ldg(plane + oy[ty]);
          p = fmaf(P, wy[ty], p);
          py = fmaf(P, dy[ty], py);
        }
        phi = fmaf(wx, p, phi);
        gx = fmaf(dx, p, gx);
        gy = fmaf(wx, py, gy);
      }
      const float wz = sW[wp][j][2][g];
      gz = phi * sD[wp][j][2][g];
      phi *= wz;
      gx *= wz;
      gy *= wz;
    }
#pragma unroll
    for (int q = 4; q > 0; q >>= 1) {
      phi += __shfl_xor_sync(kFull, phi, q);
      gx += __shfl_xor_sync(kFull, gx, q);
      gy += __shfl_xor_sync(kFull, gy, q);
      gz += __shfl_xor_sync(kFull, gz, q);
    }
    if (valid && g < 3) {  // lane g: component g
      const RepInfo &ri = a.rep[r];
      const float c = 2.f * qe;
      float f;
      if (!a.tric) {
        f = c * (g == 0 ? gx : (g == 1 ? gy : gz)) * ((float)pr.K[g] / ri.box[g]);
      } else {  // dU/dx = H^-T dU/ds
        const RecipCell k = recip_cell(ri);
        const float hx = c * gx * (float)pr.K[0], hy = c * gy * (float)pr.K[1], hz = c * gz * (float)pr.K[2];
        f = g == 0 ? hx * k.xx : (g == 1 ? fmaf(hx, k.xy, hy * k.yy) : fmaf(hx, k.xz, fmaf(hy, k.yz, hz * k.zz)));
      }
      if (o.force64) out64(&o.force64[3 * atom + g], f, a.mode);
      if (o.force) out32(&o.force[3 * atom + g], f, a.mode);
    }
    float e = 0.f;
    if (valid && g == 0) {
      if (block) red_add(&a.accL[block], to_fix(2.f * qraw * phi));
      if (ENERGY) e = qe * phi;
    }
    if (ENERGY) {
      // one atomic per warp when its 4 atoms share a replica
      const int r0 = __shfl_sync(kFull, r, 0);
      const bool same = __all_sync(kFull, !valid || r == r0);
      long long ef = to_fix(e);
      if (same) {
#pragma unroll
        for (int o2 = 16; o2 > 0; o2 >>= 1) ef += __shfl_xor_sync(kFull, ef, o2);
        if (lane == 0 && ef) red_add(&a.accE[r0], ef);
      } else if (ef) {
        red_add(&a.accE[r], ef);
      }
    }
  }
  // without energy and MSLD atoms there is nothing to wait for: the sums are zero
  if (ENERGY || a.alch) finalize_if_last(a, o, ENERGY);
  else if (blockIdx.x == 0) finalize_outputs(a, o, false);
}

// ---------------------------------------------------------------------------
// Ewald self term: one thread per atom.
// ---------------------------------------------------------------------------
template <bool ENERGY>
__global__ void k_self(PmeArgs a, float pre, bnb_outputs o) {
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int atom = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = atom < a.N;
  float e = 0.f;
  int r = 0;
  if (valid) {
    r = a.atomRep[atom];
    int block;
    const float l = atom_scale(a, atom, block);
    const float q = a.q[atom];
    const float es = pre * q * q;
    if (block) red_add(&a.accL[block], to_fix(2.f * l * es));
    e = l * l * es;
  }
  if (ENERGY) {
    const int r0 = __shfl_sync(kFull, r, 0);
    const bool same = __all_sync(kFull, !valid || r == r0);
    long long ef = to_fix(e);
    if (same) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ef += __shfl_xor_sync(kFull, ef, o);
      if (lane == 0 && ef) red_add(&a.accE[r0], ef);
    } else if (ef) {
      red_add(&a.accE[r], ef);
    }
  }
  finalize_if_last(a, o, ENERGY);
}

// lambda and energy accumulators -> outputs when there are no atoms (one CTA).
__global__ void k_pme_finalize(PmeArgs a, bnb_outputs o, bool energy) {
  pdl_wait();
  finalize_outputs(a, o, energy);
}

inline int grid_of(long long threads, int block) {
  long long g = (threads + block - 1) / block;
  return (int)(g < 1 ? 1 : (g > 148LL * 64 ? 148LL * 64 : g));
}

}  // namespace

int pme_spread(const PmeArgs &a, cudaStream_t s) {
  if (a.N > 0) {
    // 9 atoms a warp, or 3 while those would leave SMs without a CTA (gather: 8 or
    // 4): 648 atoms 29.9 -> 23.3 us an evaluation
    const bool few = a.N < 148 * 8 * kSpreadAtoms;
    const int per = few ? 3 : kSpreadAtoms, grid = (a.N + 8 * per - 1) / (8 * per);
    switch (a.order * 2 + few) {
      case 8: launch_pdl(k_spread<4, false>, grid, 256, 0, s, a); break;
      case 9: launch_pdl(k_spread<4, true>, grid, 256, 0, s, a); break;
      case 12: launch_pdl(k_spread<6, false>, grid, 256, 0, s, a); break;
      case 13: launch_pdl(k_spread<6, true>, grid, 256, 0, s, a); break;
      case 16: launch_pdl(k_spread<8, false>, grid, 256, 0, s, a); break;
      case 17: launch_pdl(k_spread<8, true>, grid, 256, 0, s, a); break;
      default: return BNB_ERR_ARG;
    }
  }
  return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_CUDA;
}

int pme_to_grid(const PmeArgs &a, cudaStream_t s) {
  launch_pdl(k_fix_to_grid, grid_of(a.totalGrid, 256), 256, 0, s, a);
  return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_CUDA;
}

int pme_convolve(const PmeArgs &a, cudaStream_t s) {
  int gx = (a.maxCplx + 1023) / 1024;  // about 4 elements per thread
  gx = gx < 1 ? 1 : gx;
  launch_pdl(k_convolve, dim3(gx, a.R), 256, 0, s, a);
  return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_CUDA;
}

int pme_gather(const PmeArgs &a, const bnb_outputs &o, bool energy, cudaStream_t s) {
  if (a.N > 0) {
    const bool few = a.N < 148 * 8 * kGatherAtoms;
    const int per = few ? 4 : kGatherAtoms, grid = (a.N + 8 * per - 1) / (8 * per);
    switch (a.order * 4 + (energy ? 2 : 0) + few) {
      case 16: launch_pdl(k_gather<4, false, false>, grid, 256, 0, s, a, o); break;
      case 17: launch_pdl(k_gather<4, false, true>, grid, 256, 0, s, a, o); break;
      case 18: launch_pdl(k_gather<4, true, false>, grid, 256, 0, s, a, o); break;
      case 19: launch_pdl(k_gather<4, true, true>, grid, 256, 0, s, a, o); break;
      case 24: launch_pdl(k_gather<6, false, false>, grid, 256, 0, s, a, o); break;
      case 25: launch_pdl(k_gather<6, false, true>, grid, 256, 0, s, a, o); break;
      case 26: launch_pdl(k_gather<6, true, false>, grid, 256, 0, s, a, o); break;
      case 27: launch_pdl(k_gather<6, true, true>, grid, 256, 0, s, a, o); break;
      case 32: launch_pdl(k_gather<8, false, false>, grid, 256, 0, s, a, o); break;
      case 33: launch_pdl(k_gather<8, false, true>, grid, 256, 0, s, a, o); break;
      case 34: launch_pdl(k_gather<8, true, false>, grid, 256, 0, s, a, o); break;
      case 35: launch_pdl(k_gather<8, true, true>, grid, 256, 0, s, a, o); break;
      default: return BNB_ERR_ARG;
    }
  } else {
    launch_pdl(k_pme_finalize, 1, 256, 0, s, a, o, energy);
  }
  return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_CUDA;
}

int pme_self(const PmeArgs &a, const bnb_outputs &o, bool energy, cudaStream_t s) {
  // -beta / sqrt(pi) (kElectric is inside the scaled charges)
  const float pre = (float)(-(double)a.beta / sqrt(kPi));
  if (a.N > 0) {
    const int grid = (a.N + 255) / 256;
    if (energy) launch_pdl(k_self<true>, grid, 256, 0, s, a, pre, o);
    else launch_pdl(k_self<false>, grid, 256, 0, s, a, pre, o);
  } else {
    launch_pdl(k_pme_finalize, 1, 256, 0, s, a, o, energy);
  }
  return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_CUDA;
}

}  // namespace bnb
