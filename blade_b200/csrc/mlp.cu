// BF16 multilayer perceptron kernels for learned landscape flattening (sm_100a).
//
// No reference counterpart: BLaDE's src/mlp is TorchANI inference through
// LibTorch, unrelated to lambda biases.  The network maps lambda histograms
// and the current bias parameters to corrections of those parameters; it is
// trained and run with these kernels only:
//   linear forward   Z = X W^T + b, Y = act(Z)  (X, W, Y in BF16; Z FP32)
//   linear backward  dZ = dY act'(Z); dX = dZ W; dW = dZ^T X; db = sum_m dZ
//   MSE loss         L = (1/M) sum_m sum_n w_n w_mn (Y - T)^2, dY = dL/dY
//   Adam             FP32 master weights, BF16 working copy
// Every product takes BF16 operands (round to nearest even) and accumulates
// in FP32 in a fixed order on the tensor pipe (mma.sync m16n8k16), so results
// are reproducible run to run.  act is
// 0 (identity) or 1 (SiLU, z * sigmoid(z)).
// All kernels are launched with programmatic dependent launch: at these sizes
// a launch's latency is as long as its work.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "bnb.h"
#include "bnb_internal.h"

namespace cg = cooperative_groups;
using bnb::ClusterGrid;
using bnb::launch_pdl;
using bnb::pdl_wait;

namespace {

__device__ __forceinline__ uint16_t f2bf(float f) {
  __nv_bfloat16 h = __float2bfloat16_rn(f);
  return *reinterpret_cast<uint16_t *>(&h);
}
__device__ __forceinline__ float sigmoid(float z) { return 1.f / (1.f + expf(-z)); }

// ---------------------------------------------------------------------------
// Products C[i,j] = sum_l A(i,l) B(l,j) over dense BF16 operands.
//
// Each operand is stored with either the sum index l contiguous (A row-major
// [I,L], B as [J,L]) or its own index contiguous (A as [L,I], B as [L,J]); it
// is staged in shared memory as it is stored, and ldmatrix (.trans for the
// second form) makes the fragments, so the forward product and both backward
// products run through one kernel without a transposition.
//
// What bounds it: the network's products (256 x 256 x 1664 and smaller) hold
// 0.01-0.2 GFLOP each, so a product lasts as long as the memory latencies one
// CTA sees in a row.  Hence: T x T output tiles with T = 32 unless 64 still
// gives half the SMs a tile, l in chunks of 64 through a ring of cp.async
// buffers (7 chunks in flight at T = 32), and two products that do not depend
// on one another (dW and dX) in one launch.  l is not split over CTAs: each
// element is one chain of k16 steps in increasing order, so every result,
// and with it every BF16 rounding downstream, is that of any other tiling.
// Measured (B200, network 1664-256-256-256-128): a training step of batch 256
// 487 -> 102 us, a forward pass of a small batch 215 -> 32 us against 64 x 64
// tiles staged element by element without overlap (11 products of 52 us each),
// separate bias/activation, column-sum and per-tensor Adam launches.
// ---------------------------------------------------------------------------
constexpr int kC = 64;       // l per chunk

struct Product {
  const uint16_t *A, *B;
  int I, J, L;
  int lastA, lastB;   // 1: the operand's own index is contiguous (A as [L,I], B as [L,J])
  int tilesJ, tiles;  // T x T output tiles
  float *C;           // [I,J]
  const float *bias;  // [J] or null
  int act;            // forward only (Y or Yf set): 0 identity, 1 SiLU
  uint16_t *Y;        // [I,J] BF16 of act(C + bias), or null
  float *Yf;          // the same in FP32, or null
};
struct Products {
  Product p[2];
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool in) {
  const int n = in ? 16 : 0;  // 0 source bytes: the 16 are zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n));
}
__device__ __forceinline__ void ldsm4(uint32_t addr, bool trans, uint32_t (&r)[4]) {
  if (trans)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Shared-memory pitch (elements) of a staged operand: [T][kC] or [kC][T].  Both
// pitches are odd multiples of 16 bytes, so the 8 rows of an ldmatrix matrix
// fall into different banks.
template <int T>
__device__ __forceinline__ int pitch_of(bool last) {
  return last ? T + 8 : kC + 8;
}
template <int T>
constexpr int stages() {  // ring of chunks: 80 KB (T = 32) or 72 KB (T = 64) of shared memory
  return T == 32 ? 8 : 4;
}
template <int T>
constexpr int stage_elems() {
  return T * (kC + 8) > kC * (T + 8) ? T * (kC + 8) : kC * (T + 8);
}

// Stages rows r0.. (own index) x l0.. of one operand; `last` as in Product.
// VEC: 16-byte asynchronous copies (the contiguous extent is a multiple of 8
// elements and the base 16-byte aligned, so a copy lies inside or outside as a
// whole); otherwise element by element.
template <int T, int THREADS, bool VEC>
__device__ __forceinline__ void stage(uint16_t *dst, const uint16_t *src, int R, int L, bool last, int r0, int l0) {
  const int pitch = pitch_of<T>(last);
  if (VEC) {
    const int cpr = last ? T / 8 : kC / 8;  // copies per staged row
#pragma unroll
    for (int c = threadIdx.x; c < T * kC / 8; c += THREADS) {
      const int row = c / cpr, col = (c - row * cpr) * 8;
      const int r = r0 + (last ? col : row), l = l0 + (last ? row : col);
      const bool in = r < R && l < L;
      const size_t at = last ? (size_t)l * R + r : (size_t)r * L + l;
      cp_async16(smem_u32(dst + row * pitch + col), in ? src + at : src, in);
    }
  } else {
    // eight loads in flight: one at a time, each behind a division, a training step
    // of a 101-33-5 network at batch 4,096 took 645 us, so 455
    constexpr int kBatch = 8;
    static_assert(T * kC % (kBatch * THREADS) == 0, "whole batches");
    const int shift = last && T == 32 ? 5 : 6, w = 1 << shift;  // T or kC elements a staged row
#pragma unroll 1
    for (int c0 = threadIdx.x; c0 < T * kC; c0 += kBatch * THREADS) {
      uint16_t v[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; k++) {
        const int c = c0 + k * THREADS, row = c >> shift, col = c & (w - 1);
        const int r = r0 + (last ? col : row), l = l0 + (last ? row : col);
        v[k] = r < R && l < L ? src[last ? (size_t)l * R + r : (size_t)r * L + l] : (uint16_t)0;
      }
#pragma unroll
      for (int k = 0; k < kBatch; k++) {
        const int c = c0 + k * THREADS;
        dst[(c >> shift) * pitch + (c & (w - 1))] = v[k];
      }
    }
  }
}

// T = 64: 2 x 4 warps of 32 x 16; T = 32: 2 x 2 warps of 16 x 16.
template <int T, bool VEC>
__global__ void __launch_bounds__(T == 64 ? 256 : 128) k_gemm_bf16(Products ps) {
  pdl_wait();
  constexpr int THREADS = T == 64 ? 256 : 128;
  constexpr int WN = T / 16;      // warps along j
  constexpr int MT = T / 32;      // 16-row fragments per warp (2 warps along i)
  constexpr int STAGE = stage_elems<T>(), kStages = stages<T>();
  extern __shared__ __align__(16) uint16_t sm[];
  const Product &p = blockIdx.x < ps.p[0].tiles ? ps.p[0] : ps.p[1];
  const int tile = blockIdx.x < ps.p[0].tiles ? blockIdx.x : blockIdx.x - ps.p[0].tiles;
  const int i0 = tile / p.tilesJ * T, j0 = tile % p.tilesJ * T;
  const bool tA = p.lastA != 0, tB = p.lastB != 0;
  const int pA = pitch_of<T>(tA), pB = pitch_of<T>(tB);
  const int n = (p.L + kC - 1) / kC;  // chunks of l

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wm = warp / WN * (MT * 16), wn = warp % WN * 16;  // warp's corner in the tile
  const int mat = lane >> 3, r8 = lane & 7;
  // element offsets of this lane's ldmatrix rows inside a stage, at k = 0
  const int aoff = tA ? ((mat >> 1) * 8 + r8) * pA + wm + (mat & 1) * 8 : (wm + (mat & 1) * 8 + r8) * pA + (mat >> 1) * 8;
  const int astep = tA ? 16 * pA : 16, arow = tA ? 16 : 16 * pA;
  const int boff = tB ? ((mat & 1) * 8 + r8) * pB + wn + (mat >> 1) * 8 : (wn + (mat >> 1) * 8 + r8) * pB + (mat & 1) * 8;
  const int bstep = tB ? 16 * pB : 16;

  float acc[MT][2][4] = {};
  auto load = [&](int c) {
    if (c < n) {
      uint16_t *s = sm + (c % kStages) * 2 * STAGE;
      stage<T, THREADS, VEC>(s, p.A, p.I, p.L, tA, i0, c * kC);
      stage<T, THREADS, VEC>(s + STAGE, p.B, p.J, p.L, tB, j0, c * kC);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
#pragma unroll
  for (int c = 0; c < kStages - 1; c++) load(c);
  for (int c = 0; c < n; c++) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kStages - 2) : "memory");
    __syncthreads();  // chunk c is staged, and every warp is done with the buffer refilled next
    load(c + kStages - 1);
    const uint16_t *s = sm + (c % kStages) * 2 * STAGE;
    const uint32_t aA = smem_u32(s + aoff), aB = smem_u32(s + STAGE + boff);
#pragma unroll
    for (int k = 0; k < kC / 16; k++) {
      uint32_t a[MT][4], b[4];
#pragma unroll
      for (int m = 0; m < MT; m++) ldsm4(aA + 2 * (k * astep + m * arow), tA, a[m]);
      ldsm4(aB + 2 * k * bstep, tB, b);
#pragma unroll
      for (int m = 0; m < MT; m++) {
        mma_bf16_16816(acc[m][0], a[m], b[0], b[1]);
        mma_bf16_16816(acc[m][1], a[m], b[2], b[3]);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  // the tile through shared memory, for whole-row stores
  constexpr int PT = T + 4;
  float *part = reinterpret_cast<float *>(sm);
#pragma unroll
  for (int m = 0; m < MT; m++)
#pragma unroll
    for (int q = 0; q < 2; q++)
#pragma unroll
      for (int h = 0; h < 2; h++)
        *reinterpret_cast<float2 *>(&part[(wm + 16 * m + 8 * h + (lane >> 2)) * PT + wn + 8 * q + 2 * (lane & 3)]) =
            make_float2(acc[m][q][2 * h], acc[m][q][2 * h + 1]);
  __syncthreads();
  if (VEC && (p.J & 3) == 0) {
    for (int e = threadIdx.x; e < T * T / 4; e += THREADS) {
      const int r = e / (T / 4), q = (e - r * (T / 4)) * 4, i = i0 + r, j = j0 + q;
      if (i >= p.I || j >= p.J) continue;
      const size_t at = (size_t)i * p.J + j;
      const float4 v = *reinterpret_cast<const float4 *>(part + r * PT + q);
      float z[4] = {v.x, v.y, v.z, v.w}, y[4];
      if (p.bias)
        for (int k = 0; k < 4; k++) z[k] += p.bias[j + k];
#pragma unroll
      for (int k = 0; k < 4; k++) y[k] = p.act ? z[k] * sigmoid(z[k]) : z[k];
      *reinterpret_cast<float4 *>(p.C + at) = make_float4(z[0], z[1], z[2], z[3]);
      if (p.Yf) *reinterpret_cast<float4 *>(p.Yf + at) = make_float4(y[0], y[1], y[2], y[3]);
      if (p.Y)
        *reinterpret_cast<uint2 *>(p.Y + at) = make_uint2((uint32_t)f2bf(y[0]) | ((uint32_t)f2bf(y[1]) << 16),
                                                          (uint32_t)f2bf(y[2]) | ((uint32_t)f2bf(y[3]) << 16));
    }
  } else {  // a column a thread, so that a warp's stores lie side by side (forward of 101-33-5 at 65,536: 90 -> 59 us)
#pragma unroll 4
    for (int e = threadIdx.x; e < T * T; e += THREADS) {
      const int r = e / T, q = e - r * T, i = i0 + r, j = j0 + q;
      if (i >= p.I || j >= p.J) continue;
      const size_t at = (size_t)i * p.J + j;
      float z = part[r * PT + q];
      if (p.bias) z += p.bias[j];
      const float y = p.act ? z * sigmoid(z) : z;
      p.C[at] = z;
      if (p.Yf) p.Yf[at] = y;
      if (p.Y) p.Y[at] = f2bf(y);
    }
  }
}

// Y, Yf = act(Z), where the product's own epilogue may not write them.
__global__ void k_act(int n, const float *Z, int act, uint16_t *Y, float *Yf) {
  pdl_wait();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const float z = Z[t], y = act ? z * sigmoid(z) : z;
  if (Y) Y[t] = f2bf(y);
  if (Yf) Yf[t] = y;
}

// dZ = dY act'(Z): FP32 copy, BF16 copy (for the products) and its column
// sums db[n] = sum_m dZ[m,n].  A CTA owns 32 columns and takes 128 rows at a
// time with all its threads; the sum of a column is 8 slices (slice r adds
// rows r, r+8, ... in order) added in a fixed tree, so it is reproducible.
constexpr int kGradRows = 128;
__global__ void __launch_bounds__(1024) k_act_grad(int M, int N, const float *dY, const float *Z, int act, float *dZ,
                                                   uint16_t *dZb, float *db) {
  pdl_wait();
  __shared__ float tile[kGradRows][33];
  __shared__ float part[8][33];
  const int c = threadIdx.x & 31, r = threadIdx.x >> 5;
  const int n = blockIdx.x * 32 + c;
  float s = 0.f;
  for (int m0 = 0; m0 < M; m0 += kGradRows) {
#pragma unroll
    for (int k = 0; k < kGradRows / 32; k++) {
      const int row = r + 32 * k, m = m0 + row;
      if (n < N && m < M) {
        const size_t t = (size_t)m * N + n;
        float g = dY[t];
        if (act) {
          const float z = Z[t], sg = sigmoid(z);
          g *= sg * (1.f + z * (1.f - sg));
        }
        dZ[t] = g;
        dZb[t] = f2bf(g);
        tile[row][c] = g;
      }
    }
    __syncthreads();
    const int rows = M - m0 < kGradRows ? M - m0 : kGradRows;
    if (r < 8 && n < N)
      for (int row = r; row < rows; row += 8) s += tile[row][c];
    __syncthreads();
  }
  if (r < 8) part[r][c] = s;
  __syncthreads();
  if (r == 0 && n < N)
    db[n] = ((part[0][c] + part[1][c]) + (part[2][c] + part[3][c])) +
            ((part[4][c] + part[5][c]) + (part[6][c] + part[7][c]));
}

// Loss and dY of the weighted mean squared error: one cluster of 8 CTAs, each
// thread's terms, the threads of a CTA and the CTAs added in a fixed order.
constexpr int kMseCtas = 8;
__global__ void __launch_bounds__(1024) k_mse(int M, int N, const float *Y, const float *T, const float *w,
                                              const float *we, float *dY, double *loss) {
  pdl_wait();
  __shared__ double red[33];
  const float inv = 1.f / (float)M;
  const int n = M * N;
  double s = 0.0;
  for (int t = blockIdx.z * 1024 + threadIdx.x; t < n; t += kMseCtas * 1024) {
    const float wn = (w ? w[t % N] : 1.f) * (we ? we[t] : 1.f);
    const float d = Y[t] - T[t];
    dY[t] = 2.f * wn * d * inv;
    s += (double)wn * d * d;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = red[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
    if (threadIdx.x == 0) red[32] = s;
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  if (blockIdx.z == 0 && threadIdx.x == 0 && loss) {
    double a = 0.0;
    for (int k = 0; k < kMseCtas; k++) a += *cluster.map_shared_rank(&red[32], k);
    *loss = a / M;
  }
  cluster.sync();
}

__device__ __forceinline__ float adam_one(float w, float gt, float &m, float &v, float lr, float b1, float b2,
                                          float eps, float wd, float c1, float c2) {
  m = b1 * m + (1.f - b1) * gt;
  v = b2 * v + (1.f - b2) * gt * gt;
  return w - lr * ((m / c1) / (sqrtf(v / c2) + eps) + wd * w);
}

// VEC: four parameters per thread (n a multiple of 4, all arrays aligned).
template <bool VEC>
__global__ void k_adam(int n, float *master, uint16_t *wb, const float *g, float *m, float *v, float lr, float b1,
                       float b2, float eps, float wd, float c1, float c2) {
  pdl_wait();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (VEC) {
    if (4 * (long long)t >= n) return;
    float4 w4 = reinterpret_cast<float4 *>(master)[t], m4 = reinterpret_cast<float4 *>(m)[t];
    float4 v4 = reinterpret_cast<float4 *>(v)[t];
    const float4 g4 = reinterpret_cast<const float4 *>(g)[t];
    w4.x = adam_one(w4.x, g4.x, m4.x, v4.x, lr, b1, b2, eps, wd, c1, c2);
    w4.y = adam_one(w4.y, g4.y, m4.y, v4.y, lr, b1, b2, eps, wd, c1, c2);
    w4.z = adam_one(w4.z, g4.z, m4.z, v4.z, lr, b1, b2, eps, wd, c1, c2);
    w4.w = adam_one(w4.w, g4.w, m4.w, v4.w, lr, b1, b2, eps, wd, c1, c2);
    reinterpret_cast<float4 *>(m)[t] = m4;
    reinterpret_cast<float4 *>(v)[t] = v4;
    reinterpret_cast<float4 *>(master)[t] = w4;
    if (wb)
      reinterpret_cast<uint2 *>(wb)[t] = make_uint2((uint32_t)f2bf(w4.x) | ((uint32_t)f2bf(w4.y) << 16),
                                                    (uint32_t)f2bf(w4.z) | ((uint32_t)f2bf(w4.w) << 16));
  } else {
    if (t >= n) return;
    float mt = m[t], vt = v[t];
    const float w = adam_one(master[t], g[t], mt, vt, lr, b1, b2, eps, wd, c1, c2);
    m[t] = mt;
    v[t] = vt;
    master[t] = w;
    if (wb) wb[t] = f2bf(w);
  }
}

template <bool VEC>
__global__ void k_to_bf16(int n, const float *x, uint16_t *y) {
  pdl_wait();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (VEC) {
    if (4 * (long long)t >= n) return;
    const float4 v = reinterpret_cast<const float4 *>(x)[t];
    reinterpret_cast<uint2 *>(y)[t] = make_uint2((uint32_t)f2bf(v.x) | ((uint32_t)f2bf(v.y) << 16),
                                                 (uint32_t)f2bf(v.z) | ((uint32_t)f2bf(v.w) << 16));
  } else if (t < n) {
    y[t] = f2bf(x[t]);
  }
}

inline int grid1(long long n) { return (int)((n + 255) / 256); }
// Whether a bytes from p and b bytes from q share memory (null: no).
inline bool overlap(const void *p, size_t a, const void *q, size_t b) {
  const uintptr_t x = reinterpret_cast<uintptr_t>(p), y = reinterpret_cast<uintptr_t>(q);
  return x && y && x < y + b && y < x + a;
}
inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
inline bool aligned8(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 7) == 0; }

template <int T, bool VEC>
int gemm_t(Products &ps, int count, cudaStream_t s) {
  constexpr size_t smem = sizeof(uint16_t) * 2 * stages<T>() * stage_elems<T>();
  static_assert(smem >= sizeof(float) * T * (T + 4), "the tile fits the staging buffers");
  int tiles = 0;
  for (int k = 0; k < 2; k++) {
    Product &p = ps.p[k];
    if (k >= count) {
      p = ps.p[0];
      p.tiles = 0;
      continue;
    }
    p.tilesJ = (p.J + T - 1) / T;
    p.tiles = (p.I + T - 1) / T * p.tilesJ;
    tiles += p.tiles;
  }
  auto k = k_gemm_bf16<T, VEC>;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return BNB_ERR_CUDA;
  launch_pdl(k, tiles, T == 64 ? 256 : 128, smem, s, ps);
  return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_CUDA;
}

int gemm(Products &ps, int count, cudaStream_t s) {
  long long tiles64 = 0;
  bool vec = true;
  for (int k = 0; k < count; k++) {
    const Product &p = ps.p[k];
    tiles64 += (long long)((p.I + 63) / 64) * ((p.J + 63) / 64);
    vec = vec && (p.lastA ? p.I : p.L) % 8 == 0 && (p.lastB ? p.J : p.L) % 8 == 0 && aligned16(p.A) &&
          aligned16(p.B) && aligned16(p.C) && aligned16(p.Yf) && aligned8(p.Y);
  }
  if (tiles64 >= 74) return vec ? gemm_t<64, true>(ps, count, s) : gemm_t<64, false>(ps, count, s);
  return vec ? gemm_t<32, true>(ps, count, s) : gemm_t<32, false>(ps, count, s);
}

}  // namespace

extern "C" int bnb_mlp_linear_forward(int M, int N, int K, const uint16_t *X, const uint16_t *W, const float *bias,
                                      int act, float *Z, uint16_t *Y, float *Yf, void *stream) {
  if (M < 0 || N < 0 || K < 0 || !X || !W || !Z || (act != 0 && act != 1)) return BNB_ERR_ARG;
  if ((long long)M * N >= (1ll << 31)) return BNB_ERR_ARG;
  if (M == 0 || N == 0) return BNB_OK;
  // A layer in place (Y over X): other tiles still read the inputs while one writes
  // its outputs, so the activation is a launch of its own.
  const size_t n = (size_t)M * N, k2 = 2 * (size_t)K;
  const bool apart = !overlap(Y, 2 * n, X, M * k2) && !overlap(Yf, 4 * n, X, M * k2) && !overlap(Y, 2 * n, W, N * k2) &&
                     !overlap(Yf, 4 * n, W, N * k2) && !overlap(Y, 2 * n, bias, 4 * (size_t)N) &&
                     !overlap(Yf, 4 * n, bias, 4 * (size_t)N);
  Products ps{};
  // Z[m,n] = sum_k X[m,k] W[n,k]
  ps.p[0] = Product{X, W, M, N, K, 0, 0, 0, 0, Z, bias, act, apart ? Y : nullptr, apart ? Yf : nullptr};
  const int rc = gemm(ps, 1, (cudaStream_t)stream);
  if (rc || apart) return rc;
  launch_pdl(k_act, grid1((long long)n), 256, 0, (cudaStream_t)stream, (int)n, Z, act, Y, Yf);
  return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_CUDA;
}

extern "C" int bnb_mlp_linear_backward(int M, int N, int K, const float *dY, const float *Z, int act,
                                       const uint16_t *X, const uint16_t *W, float *dZ, uint16_t *dZb, float *dX,
                                       float *dW, float *db, void *stream) {
  if (M < 0 || N < 0 || K < 0 || !dY || !Z || !X || !W || !dZ || !dZb || !dW || !db || (act != 0 && act != 1))
    return BNB_ERR_ARG;
  if ((long long)M * N >= (1ll << 31) || (long long)M * K >= (1ll << 31)) return BNB_ERR_ARG;
  if (M == 0 || N == 0) return BNB_OK;
  cudaStream_t s = (cudaStream_t)stream;
  launch_pdl(k_act_grad, (N + 31) / 32, 1024, 0, s, M, N, dY, Z, act, dZ, dZb, db);
  if (cudaGetLastError() != cudaSuccess) return BNB_ERR_CUDA;
  if (K == 0) return BNB_OK;
  // dW[n,k] = sum_m dZ[m,n] X[m,k], dX[m,k] = sum_n dZ[m,n] W[n,k]
  const Product w{dZb, X, N, K, M, 1, 1, 0, 0, dW, nullptr, 0, nullptr, nullptr};
  const Product x{dZb, W, M, K, N, 0, 1, 0, 0, dX, nullptr, 0, nullptr, nullptr};
  Products both{{w, x}};
  if (!dX || !overlap(dX, 4 * (size_t)M * K, X, 2 * (size_t)M * K)) return gemm(both, dX ? 2 : 1, s);
  // dX over X, which dW reads first
  Products first{{w, w}}, second{{x, x}};
  const int rc = gemm(first, 1, s);
  return rc ? rc : gemm(second, 1, s);
}

extern "C" int bnb_mlp_mse(int M, int N, const float *Y, const float *T, const float *weight,
                           const float *elemWeight, float *dY, double *loss, void *stream) {
  if (M <= 0 || N <= 0 || !Y || !T || !dY) return BNB_ERR_ARG;
  launch_pdl(k_mse, ClusterGrid{dim3(1, 1, kMseCtas), kMseCtas}, 1024, 0, (cudaStream_t)stream, M, N, Y, T, weight,
             elemWeight, dY, loss);
  return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_CUDA;
}

extern "C" int bnb_mlp_adam(int n, float *master, uint16_t *weightBf16, const float *grad, float *m, float *v,
                            float lr, float beta1, float beta2, float eps, float weightDecay, int step,
                            void *stream) {
  if (n < 0 || step < 1 || (n > 0 && (!master || !grad || !m || !v))) return BNB_ERR_ARG;
  if (n == 0) return BNB_OK;
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  const bool vec = n % 4 == 0 && aligned16(master) && aligned16(grad) && aligned16(m) && aligned16(v) &&
                   aligned8(weightBf16);
  if (vec)
    launch_pdl(k_adam<true>, grid1(n / 4), 256, 0, (cudaStream_t)stream, n, master, weightBf16, grad, m, v, lr, beta1,
               beta2, eps, weightDecay, c1, c2);
  else
    launch_pdl(k_adam<false>, grid1(n), 256, 0, (cudaStream_t)stream, n, master, weightBf16, grad, m, v, lr, beta1,
               beta2, eps, weightDecay, c1, c2);
  return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_CUDA;
}

extern "C" int bnb_to_bf16(int n, const float *x, uint16_t *y, void *stream) {
  if (n < 0 || (n > 0 && (!x || !y))) return BNB_ERR_ARG;
  if (n == 0) return BNB_OK;
  if (n % 4 == 0 && aligned16(x) && aligned8(y))
    launch_pdl(k_to_bf16<true>, grid1(n / 4), 256, 0, (cudaStream_t)stream, n, x, y);
  else
    launch_pdl(k_to_bf16<false>, grid1(n), 256, 0, (cudaStream_t)stream, n, x, y);
  return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_CUDA;
}
