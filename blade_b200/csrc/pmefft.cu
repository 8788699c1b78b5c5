// 3-D transforms of the PME grids (sm_100a): three launches for all replicas
// and grid sizes instead of a cuFFT plan (three launches each way) per size.
//
//   k_pme_plane_forward  one CTA per x plane: charge grid (fixed point, cleared
//                        for the next call) -> real transforms along z, two
//                        rows as one complex sequence -> transforms along y
//   k_pme_x              a tile of (y, z) columns per CTA: transform along x,
//                        influence function, inverse transform along x
//   k_pme_plane_inverse  one CTA per x plane: inverse along y and z
//
// The transforms are Stockham autosort passes (radices 2-6 and 8, any length
// that they factor) between two shared-memory buffers, FP32 with twiddles
// rounded from FP64.  What bounds them at these sizes (32^3 to 128^3, all in
// L2) is the number of launches and the synchronised passes in a row, not
// traffic: 64^3 takes 2 passes per direction, 128^3 three.  Measured against the
// cuFFT path (conversion, three kernels each way, convolution), one evaluation
// at order 6: 20^3 41 -> 25 us, 64^3 57 -> 47, 128^3 207 -> 196, and a step of 8
// replicas with six grid sizes 437 -> 359 us; where cuFFT is the faster is said at
// the choice in bnb_set_pme.
#include <cuda_runtime.h>

#include "pme.h"

namespace bnb {
namespace {

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 w) {
  return make_float2(fmaf(a.x, w.x, -a.y * w.y), fmaf(a.x, w.y, a.y * w.x));
}
__device__ __forceinline__ float2 mul_mi(float2 a) { return make_float2(a.y, -a.x); }  // -i a

// b_j = sum_k a_k exp(-2 pi i j k / R), in place.
template <int R>
__device__ __forceinline__ void dft(float2 (&a)[R]);
template <>
__device__ __forceinline__ void dft<2>(float2 (&a)[2]) {
  const float2 t = a[0];
  a[0] = cadd(t, a[1]);
  a[1] = csub(t, a[1]);
}
template <>
__device__ __forceinline__ void dft<3>(float2 (&a)[3]) {
  const float2 s = cadd(a[1], a[2]), d = csub(a[1], a[2]);
  constexpr float kS = 0.86602540378443864676f;  // sin(pi/3)
  const float2 m = make_float2(fmaf(-0.5f, s.x, a[0].x), fmaf(-0.5f, s.y, a[0].y));
  const float2 e = make_float2(kS * d.y, -kS * d.x);  // -i sin d
  a[0] = cadd(a[0], s);
  a[1] = cadd(m, e);
  a[2] = csub(m, e);
}
template <>
__device__ __forceinline__ void dft<4>(float2 (&a)[4]) {
  const float2 s0 = cadd(a[0], a[2]), d0 = csub(a[0], a[2]), s1 = cadd(a[1], a[3]), d1 = mul_mi(csub(a[1], a[3]));
  a[0] = cadd(s0, s1);
  a[1] = cadd(d0, d1);
  a[2] = csub(s0, s1);
  a[3] = csub(d0, d1);
}
template <>
__device__ __forceinline__ void dft<5>(float2 (&a)[5]) {
  constexpr float c1 = 0.30901699437494742410f, c2 = -0.80901699437494742410f;  // cos(2 pi/5), cos(4 pi/5)
  constexpr float n1 = 0.95105651629515357212f, n2 = 0.58778525229247312917f;   // sin(2 pi/5), sin(4 pi/5)
  const float2 s1 = cadd(a[1], a[4]), d1 = csub(a[1], a[4]), s2 = cadd(a[2], a[3]), d2 = csub(a[2], a[3]);
  const float2 m1 = make_float2(fmaf(c1, s1.x, fmaf(c2, s2.x, a[0].x)), fmaf(c1, s1.y, fmaf(c2, s2.y, a[0].y)));
  const float2 m2 = make_float2(fmaf(c2, s1.x, fmaf(c1, s2.x, a[0].x)), fmaf(c2, s1.y, fmaf(c1, s2.y, a[0].y)));
  const float2 e1 = mul_mi(make_float2(fmaf(n1, d1.x, n2 * d2.x), fmaf(n1, d1.y, n2 * d2.y)));
  const float2 e2 = mul_mi(make_float2(fmaf(n2, d1.x, -n1 * d2.x), fmaf(n2, d1.y, -n1 * d2.y)));
  a[0] = cadd(a[0], cadd(s1, s2));
  a[1] = cadd(m1, e1);
  a[2] = cadd(m2, e2);
  a[3] = csub(m2, e2);
  a[4] = csub(m1, e1);
}
template <>
__device__ __forceinline__ void dft<6>(float2 (&a)[6]) {
  // k = 3 k1 + 2 k2 (mod 6), j with j mod 2 and j mod 3: no twiddles between
  float2 u[3] = {a[0], a[2], a[4]}, v[3] = {a[3], a[5], a[1]};
  dft<3>(u);
  dft<3>(v);
  a[0] = cadd(u[0], v[0]);
  a[3] = csub(u[0], v[0]);
  a[4] = cadd(u[1], v[1]);
  a[1] = csub(u[1], v[1]);
  a[2] = cadd(u[2], v[2]);
  a[5] = csub(u[2], v[2]);
}
template <>
__device__ __forceinline__ void dft<8>(float2 (&a)[8]) {
  float2 e[4] = {a[0], a[2], a[4], a[6]}, o[4] = {a[1], a[3], a[5], a[7]};
  dft<4>(e);
  dft<4>(o);
  constexpr float kH = 0.70710678118654752440f;
  o[1] = make_float2(kH * (o[1].x + o[1].y), kH * (o[1].y - o[1].x));
  o[2] = mul_mi(o[2]);
  o[3] = make_float2(kH * (o[3].y - o[3].x), -kH * (o[3].x + o[3].y));
#pragma unroll
  for (int k = 0; k < 4; k++) {
    a[k] = cadd(e[k], o[k]);
    a[k + 4] = csub(e[k], o[k]);
  }
}

// Quotient i / n for 0 <= i < 2^16, 1 <= n: inv = 1 / n in FP32 is off by at most
// 2^-24 relative, i + 0.5 lies at least 0.5 / n from a multiple.
__device__ __forceinline__ int quotient(int i, float inv) { return (int)(((float)i + 0.5f) * inv); }

// One Stockham pass over B interleaved sequences (element n of sequence b at
// n * pitch + b): s is the product of the radices before it.
template <int R>
__device__ __forceinline__ void pass(const float2 *in, float2 *out, int N, int s, int B, int pitch, const float2 *tw) {
  const int q = N / R, total = q * B;
  const float invB = 1.f / (float)B, invS = 1.f / (float)s;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int t = quotient(i, invB), b = i - t * B;
    const int ps = quotient(t, invS) * s;  // p s with t = p s + (t mod s)
    float2 a[R];
#pragma unroll
    for (int k = 0; k < R; k++) a[k] = in[(t + k * q) * pitch + b];
    dft<R>(a);
    float2 *o = out + (t + ps * (R - 1)) * pitch + b;
    o[0] = a[0];
#pragma unroll
    for (int j = 1; j < R; j++) o[j * s * pitch] = cmul(a[j], tw[j * ps]);
  }
}

// Forward transform of B sequences; the result is in the returned buffer.
__device__ __forceinline__ float2 *transform(float2 *x, float2 *y, int N, uint32_t plan, int B, int pitch,
                                             const float2 *tw) {
  for (int s = 1; plan; plan >>= 4) {
    const int R = plan & 15;
    switch (R) {
      case 2: pass<2>(x, y, N, s, B, pitch, tw); break;
      case 3: pass<3>(x, y, N, s, B, pitch, tw); break;
      case 4: pass<4>(x, y, N, s, B, pitch, tw); break;
      case 5: pass<5>(x, y, N, s, B, pitch, tw); break;
      case 6: pass<6>(x, y, N, s, B, pitch, tw); break;
      default: pass<8>(x, y, N, s, B, pitch, tw); break;
    }
    s *= R;
    __syncthreads();
    float2 *t = x;
    x = y;
    y = t;
  }
  return x;
}

// Shared memory: two buffers of bufElems, then the twiddle tables.
struct PlaneDims {
  int K1, K2, K2h, rows2, pitchZ, pitchY;  // rows2: pairs of rows
  __device__ __forceinline__ explicit PlaneDims(const PmeRep &p)
      : K1(p.K[1]), K2(p.K[2]), K2h(p.K[2] / 2 + 1), rows2((p.K[1] + 1) / 2), pitchZ(((p.K[1] + 1) / 2) | 1),
        pitchY((p.K[2] / 2 + 1) | 1) {}
};

__global__ void __launch_bounds__(1024) k_pme_plane_forward(PmeArgs a) {
  pdl_wait();
  extern __shared__ __align__(16) float2 fsm[];
  const int2 at = a.planeMap[blockIdx.x];  // (replica, x)
  const PmeRep pr = a.prep[at.x];
  const PlaneDims d(pr);
  float2 *x = fsm, *y = fsm + a.bufElems, *tw1 = y + a.bufElems, *tw2 = tw1 + d.K1;
  for (int i = threadIdx.x; i < d.K1; i += blockDim.x) tw1[i] = a.twiddle[pr.twOff[1] + i];
  for (int i = threadIdx.x; i < d.K2; i += blockDim.x) tw2[i] = a.twiddle[pr.twOff[2] + i];
  long long *q = a.qfix + pr.gridOff + (size_t)at.y * d.K1 * d.K2;
  const float inv2 = 1.f / (float)d.K2;
  constexpr float kUnit = (float)(1.0 / kFixScale);  // a power of two
#pragma unroll 4
  for (int i = threadIdx.x; i < d.K1 * d.K2; i += blockDim.x) {
    const long long v = q[i];
    if (v) q[i] = 0;  // ready for the next call
    const int row = quotient(i, inv2), z = i - row * d.K2;
    float2 *e = x + z * d.pitchZ + (row >> 1);
    if (row & 1) e->y = __ll2float_rn(v) * kUnit;
    else e->x = __ll2float_rn(v) * kUnit;
  }
  if (d.K1 & 1)  // the last row has no partner
    for (int z = threadIdx.x; z < d.K2; z += blockDim.x) x[z * d.pitchZ + d.rows2 - 1].y = 0.f;
  __syncthreads();
  float2 *f = transform(x, y, d.K2, pr.plan[2], d.rows2, d.pitchZ, tw2);
  float2 *h = f == x ? y : x;
  // rows 2p and 2p+1 from Z = A + i B: A[k] = (Z[k] + conj Z[K-k]) / 2, B[k] = (Z[k] - conj Z[K-k]) / 2i
  const float invH = 1.f / (float)d.K2h;
  for (int i = threadIdx.x; i < d.rows2 * d.K2h; i += blockDim.x) {
    const int p = quotient(i, invH), k = i - p * d.K2h;
    const float2 u = f[k * d.pitchZ + p], v = f[(k ? d.K2 - k : 0) * d.pitchZ + p];
    h[2 * p * d.pitchY + k] = make_float2(0.5f * (u.x + v.x), 0.5f * (u.y - v.y));
    if (2 * p + 1 < d.K1) h[(2 * p + 1) * d.pitchY + k] = make_float2(0.5f * (u.y + v.y), 0.5f * (v.x - u.x));
  }
  __syncthreads();
  const float2 *r = transform(h, f, d.K1, pr.plan[1], d.K2h, d.pitchY, tw1);
  float2 *out = a.cplx + pr.cplxOff + (size_t)at.y * d.K1 * d.K2h;
  for (int i = threadIdx.x; i < d.K1 * d.K2h; i += blockDim.x) {
    const int row = quotient(i, invH), k = i - row * d.K2h;
    out[i] = r[row * d.pitchY + k];
  }
}

__global__ void __launch_bounds__(1024) k_pme_plane_inverse(PmeArgs a) {
  pdl_wait();
  extern __shared__ __align__(16) float2 fsm[];
  const int2 at = a.planeMap[blockIdx.x];
  const PmeRep pr = a.prep[at.x];
  const PlaneDims d(pr);
  float2 *x = fsm, *y = fsm + a.bufElems, *tw1 = y + a.bufElems, *tw2 = tw1 + d.K1;
  for (int i = threadIdx.x; i < d.K1; i += blockDim.x) tw1[i] = a.twiddle[pr.twOff[1] + i];
  for (int i = threadIdx.x; i < d.K2; i += blockDim.x) tw2[i] = a.twiddle[pr.twOff[2] + i];
  // an inverse transform is a forward one with real and imaginary parts swapped before and after
  const float2 *in = a.cplx + pr.cplxOff + (size_t)at.y * d.K1 * d.K2h;
  const float invH = 1.f / (float)d.K2h, inv2 = 1.f / (float)d.K2;
#pragma unroll 4
  for (int i = threadIdx.x; i < d.K1 * d.K2h; i += blockDim.x) {
    const int row = quotient(i, invH), k = i - row * d.K2h;
    const float2 v = in[i];
    x[row * d.pitchY + k] = make_float2(v.y, v.x);
  }
  __syncthreads();
  const float2 *h = transform(x, y, d.K1, pr.plan[1], d.K2h, d.pitchY, tw1);
  float2 *z = h == x ? y : x;
  // rows A = 2p and B = 2p+1 as Z = A + i B, swapped; both are real, so Z[K-k] = conj A[k] + i conj B[k]
  for (int i = threadIdx.x; i < d.rows2 * d.K2h; i += blockDim.x) {
    const int p = quotient(i, invH), k = i - p * d.K2h;
    const float2 sa = h[2 * p * d.pitchY + k];
    const float2 sb = 2 * p + 1 < d.K1 ? h[(2 * p + 1) * d.pitchY + k] : make_float2(0.f, 0.f);
    float2 A = make_float2(sa.y, sa.x), B = make_float2(sb.y, sb.x);
    if (k == 0 || 2 * k == d.K2) A.y = B.y = 0.f;  // real by symmetry
    const float2 u = make_float2(A.x - B.y, A.y + B.x), v = make_float2(A.x + B.y, B.x - A.y);
    z[k * d.pitchZ + p] = make_float2(u.y, u.x);
    if (k && 2 * k != d.K2) z[(d.K2 - k) * d.pitchZ + p] = make_float2(v.y, v.x);
  }
  __syncthreads();
  const float2 *r = transform(z, const_cast<float2 *>(h), d.K2, pr.plan[2], d.rows2, d.pitchZ, tw2);
  float *out = a.grid + pr.gridOff + (size_t)at.y * d.K1 * d.K2;
  for (int i = threadIdx.x; i < d.K1 * d.K2; i += blockDim.x) {
    const int row = quotient(i, inv2), k = i - row * d.K2;
    const float2 v = r[k * d.pitchZ + (row >> 1)];
    out[i] = row & 1 ? v.x : v.y;  // swapped back
  }
}

// Tile of kPmeCols neighbouring columns (64 bytes of every x plane).  128 threads
// for each 160 points along x: with 128 in all, long grids had few warps to hide
// the passes' latency (an evaluation on 300 x 64 x 64 57 -> 47 us, on 600 x 64 x 64
// 84 -> 62).
__global__ void __launch_bounds__(512, 2) k_pme_x(PmeArgs a) {
  pdl_wait();
  extern __shared__ __align__(16) float2 fsm[];
  const int2 at = a.colMap[blockIdx.x];  // (replica, first column)
  const PmeRep pr = a.prep[at.x];
  const int K0 = pr.K[0], K1 = pr.K[1], K2h = pr.K[2] / 2 + 1, NC = K1 * K2h;
  const int c0 = at.y, B = NC - c0 < kPmeCols ? NC - c0 : kPmeCols;
  float2 *x = fsm, *y = fsm + K0 * kPmeCols, *tw = y + K0 * kPmeCols;
  for (int i = threadIdx.x; i < K0; i += blockDim.x) tw[i] = a.twiddle[pr.twOff[0] + i];
  float2 *spec = a.cplx + pr.cplxOff;
  const InfluenceFn fn(a, pr, a.rep[at.x]);
#pragma unroll 4
  for (int i = threadIdx.x; i < K0 * kPmeCols; i += blockDim.x) {
    const int n = i / kPmeCols, b = i % kPmeCols;
    if (b < B) x[i] = spec[(size_t)n * NC + c0 + b];
  }
  __syncthreads();
  float2 *f = transform(x, y, K0, pr.plan[0], B, kPmeCols, tw);
  float2 *g = f == x ? y : x;
  const float inv = 1.f / (float)K2h;
  for (int i = threadIdx.x; i < K0 * kPmeCols; i += blockDim.x) {
    const int n = i / kPmeCols, b = i % kPmeCols;
    if (b >= B) continue;
    const int c = c0 + b, j = quotient(c, inv), k = c - j * K2h;
    const float w = fn(n, j, k);
    const float2 v = f[i];
    f[i] = make_float2(v.y * w, v.x * w);  // swapped: the inverse transform follows
  }
  __syncthreads();
  const float2 *r = transform(f, g, K0, pr.plan[0], B, kPmeCols, tw);
  for (int i = threadIdx.x; i < K0 * kPmeCols; i += blockDim.x) {
    const int n = i / kPmeCols, b = i % kPmeCols;
    if (b < B) spec[(size_t)n * NC + c0 + b] = make_float2(r[i].y, r[i].x);
  }
}

}  // namespace

uint32_t pme_fft_plan(int n) {
  // fewest passes over the radices 8, 6, 5, 4, 3, 2, the largest first
  static const int radix[] = {8, 6, 5, 4, 3, 2};
  uint32_t best = 0;
  int bestLen = 9;
  struct Search {
    static void run(int n, int from, uint32_t plan, int len, uint32_t &best, int &bestLen) {
      if (n == 1) {
        if (len < bestLen) { best = plan; bestLen = len; }
        return;
      }
      if (len + 1 >= bestLen) return;
      for (int i = from; i < 6; i++)
        if (n % radix[i] == 0) run(n / radix[i], i, plan | ((uint32_t)radix[i] << (4 * len)), len + 1, best, bestLen);
    }
  };
  if (n > 1) Search::run(n, 0, 0, 0, best, bestLen);
  return best;  // 0: the length has another prime factor
}

size_t pme_fft_plane_smem(const int *K, int *bufElems) {
  const int z = K[2] * (((K[1] + 1) / 2) | 1), y = K[1] * ((K[2] / 2 + 1) | 1);
  *bufElems = z > y ? z : y;
  return sizeof(float2) * (2 * (size_t)*bufElems + K[1] + K[2]);
}

size_t pme_fft_x_smem(int K0) { return sizeof(float2) * ((size_t)K0 * (2 * kPmeCols + 1)); }

int pme_fft_setup() {
  // the largest any grid may ask for, so handles with different grids do not
  // take one another's setting back
  if (cudaFuncSetAttribute(k_pme_plane_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPmeFftSmem) !=
          cudaSuccess ||
      cudaFuncSetAttribute(k_pme_plane_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPmeFftSmem) !=
          cudaSuccess ||
      cudaFuncSetAttribute(k_pme_x, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPmeFftSmem) != cudaSuccess)
    return BNB_ERR_CUDA;
  return BNB_OK;
}

int pme_fft(const PmeArgs &a, const PmeFftLaunch &l, cudaStream_t s) {
  launch_pdl(k_pme_plane_forward, l.planes, l.planeThreads, l.planeSmem, s, a);
  launch_pdl(k_pme_x, l.colTiles, l.xThreads, l.xSmem, s, a);
  launch_pdl(k_pme_plane_inverse, l.planes, l.planeThreads, l.planeSmem, s, a);
  return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_CUDA;
}

}  // namespace bnb
