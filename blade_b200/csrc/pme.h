// PME reciprocal space and Ewald self term used by the C ABI layer.
#pragma once
#include <cuda_runtime.h>

#include "bnb.h"
#include "bnb_internal.h"

namespace bnb {

struct PmeRep {            // per replica: grid sizes and offsets into the concatenated grids
  int K[3];
  int gridOff;             // real grid [K0][K1][K2]
  int cplxOff;             // half spectrum [K0][K1][K2/2+1]
  int modOff;              // moduli: K0 + K1 + (K2/2+1) values
  int twOff[3];            // twiddle table of each dimension (K values), own transforms only
  uint32_t plan[3];        // radices of each dimension, 4 bits each, first pass lowest
};

constexpr int kPmeCols = 8;                   // columns per CTA of the transform along x
constexpr size_t kPmeFftSmem = 220 * 1024;    // most shared memory of a transform CTA

struct PmeArgs {
  int N, R, lamTotal, order;
  int totalGrid, totalCplx, maxCplx;  // maxCplx: largest half spectrum of one replica
  float beta, pi2Beta2;    // pi2Beta2: pi^2 / beta^2
  const float *x;          // [3N] caller positions (State::position_fd)
  const float *lambda;     // [lamTotal] or null (every scale 1)
  const float *q;          // [N] charge * sqrt(kElectric)
  const int *siteBlock;    // [N] (site<<16)|block
  const int *atomRep;      // [N]
  const RepInfo *rep;      // [R] boxes
  const PmeRep *prep;      // [R]
  const float *mod;        // moduli 1/|b(m)|^2, per replica and dimension
  long long *qfix;         // [totalGrid] fixed-point charge grid (zero between calls)
  float *grid;             // [totalGrid] charge grid, then (after C2R) the potential grid
  float2 *cplx;            // [totalCplx] spectrum
  long long *accL;         // [lamTotal]
  long long *accE;         // [R]
  unsigned int *done;      // CTAs finished in the current gather / self launch (zero between launches)
  int mode;                // BNB_OUT_SET / BNB_OUT_ADD64 bits of the call
  int alch;                // some atom belongs to an MSLD block
  int tric;                // boxes are triclinic cells (RepInfo::box and ::tric)
  // own transforms (pmefft.cu)
  const float2 *twiddle;   // exp(-2 pi i k / K) per replica and dimension
  const int2 *planeMap;    // (replica, x) of every x plane
  const int2 *colMap;      // (replica, first column) of every tile of columns
  int bufElems;            // elements of one shared-memory buffer of a plane CTA
};

struct PmeFftLaunch {
  int planes, planeThreads, colTiles, xThreads;
  size_t planeSmem, xSmem;
};

// H^-1 of a triclinic cell as (xx, xy, xz, yy, yz, zz), FP32 like the
// reference's kTricBox_f.
struct RecipCell {
  float xx, xy, xz, yy, yz, zz;
};
__device__ __forceinline__ RecipCell recip_cell(const RepInfo &ri) {
  const float ax = ri.box[0], by = ri.box[1], cz = ri.box[2];
  const float bx = ri.tric[0], cx = ri.tric[1], cy = ri.tric[2];
  const float vinv = 1.f / (ax * by * cz);
  RecipCell k;
  k.xx = by * cz * vinv;
  k.xy = -bx * cz * vinv;
  k.xz = (bx * cy - by * cx) * vinv;
  k.yy = cz * ax * vinv;
  k.yz = -cy * ax * vinv;
  k.zz = ax * by * vinv;
  return k;
}

// Influence function of a replica at spectrum element (i, j, k):
// B(m) exp(-pi^2 k^2 / beta^2) / (2 pi V k^2), FP32 like the reference's kernel
// (nbrecip.cu:215-256).
struct InfluenceFn {
  int K0, K1;
  float ix, iy, iz, c, g;
  RecipCell rc;
  bool tric;
  const float *m0, *m1, *m2;
  __device__ __forceinline__ InfluenceFn(const PmeArgs &a, const PmeRep &pr, const RepInfo &ri) {
    constexpr double pi = 3.14159265358979323846;
    K0 = pr.K[0];
    K1 = pr.K[1];
    ix = (float)ri.inv[0];
    iy = (float)ri.inv[1];
    iz = (float)ri.inv[2];
    tric = a.tric != 0;
    rc = tric ? recip_cell(ri) : RecipCell{};
    c = (float)(ri.inv[0] * ri.inv[1] * ri.inv[2] * (0.5 / pi));
    g = a.pi2Beta2;
    m0 = a.mod + pr.modOff;
    m1 = m0 + K0;
    m2 = m1 + K1;
  }
  __device__ __forceinline__ float operator()(int i, int j, int k) const {
    const float mi = (float)(2 * i <= K0 ? i : i - K0), mj = (float)(2 * j <= K1 ? j : j - K1), mk = (float)k;
    float kx, ky, kz;
    if (!tric) {
      kx = mi * ix;
      ky = mj * iy;
      kz = mk * iz;
    } else {  // k = H^-T m
      kx = mi * rc.xx;
      ky = fmaf(mi, rc.xy, mj * rc.yy);
      kz = fmaf(mi, rc.xz, fmaf(mj, rc.yz, mk * rc.zz));
    }
    const float k2 = fmaf(kx, kx, fmaf(ky, ky, kz * kz));
    return (i | j | k) == 0 ? 0.f : m0[i] * m1[j] * m2[k] * c * expf(-g * k2) / k2;
  }
};

// Radices of a transform length (PmeRep::plan), 0 if it has a prime factor above 5.
uint32_t pme_fft_plan(int n);
// Shared memory of a plane CTA (and its buffer size) and of a column CTA.
size_t pme_fft_plane_smem(const int *K, int *bufElems);
size_t pme_fft_x_smem(int K0);
int pme_fft_setup();
// qfix (cleared) -> transforms, influence function, inverse transforms ->
// potential grid; three launches.
int pme_fft(const PmeArgs &a, const PmeFftLaunch &l, cudaStream_t s);

// Spread lambda-scaled charges into qfix; one launch.
int pme_spread(const PmeArgs &a, cudaStream_t s);
// For cuFFT: qfix (cleared) -> FP32 grid; one launch.
int pme_to_grid(const PmeArgs &a, cudaStream_t s);
// Multiply the spectrum by the influence function; one launch.
int pme_convolve(const PmeArgs &a, cudaStream_t s);
// Gather forces, dU/dlambda and energy from the potential grid; the last
// CTA writes the lambda and energy outputs; one launch.
int pme_gather(const PmeArgs &a, const bnb_outputs &o, bool energy, cudaStream_t s);
// Ewald self energy and its dU/dlambda; one launch.
int pme_self(const PmeArgs &a, const bnb_outputs &o, bool energy, cudaStream_t s);

}  // namespace bnb
