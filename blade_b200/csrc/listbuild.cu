// Block neighbour-list builder for the direct-space path (sm_100a).
//
// Counterpart of the reference's Domdec::reset_domdec
// (src/domdec/domdec.cu:201-211): bin atoms into x/y columns
// (assign_blocks.cu:24-60), order each column by z (assign_blocks.cu:62-178),
// cut columns into blocks of <=32 atoms (assign_blocks.cu:189-308), build
// AABBs (assign_blocks.cu:340-382), cull block pairs over the 14-image half
// shell at rCut+pad (cull.cu:44-299) and attach 32x32 exclusion masks
// (assign_excl.cu:17-313).  Differences by design:
//   * deterministic: z ties broken by atom index; each i block's candidates
//     are in (shift code, j block) order, so the list is identical run to run
//     up to where its blocks' ranges lie in memory (bnb_get_list exports it in
//     block order);
//   * five launches: binning, column scan, scatter, one CTA per column (sort,
//     slots, packed coordinates, AABBs) and one CTA per i block (cull, exclusion
//     masks, work items);
//   * no host synchronisation: counts stay on the device and capacity
//     overflow raises a status bit instead of a host readback;
//   * batched: R replicas in one pass, tiles never cross replicas.
// Every FP32 step is one IEEE operation (__f*_rn, built with -fmad=false),
// the sequence restated on the CPU in oracle/listbuild_oracle.c.
#include <cuda_runtime.h>
#include <stdint.h>

#include "bnb_internal.h"
#include "listbuild.h"

namespace bnb {

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;

__device__ __forceinline__ uint32_t z_key(float z) {
  uint32_t u = __float_as_uint(z);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}



// AABB gap^2 <= c2 with the operation order of orc_aabb_hit.
__device__ __forceinline__ bool aabb_hit(float4 imin, float4 imax, float4 jmin,
                                         float4 jmax, float3 sh, float c2) {
  float lo, hi, g1, g2, g, acc;
  lo = __fadd_rn(jmin.x, sh.x); hi = __fadd_rn(jmax.x, sh.x);
  g1 = __fsub_rn(lo, imax.x); g2 = __fsub_rn(imin.x, hi);
  g = g1 > g2 ? g1 : g2; g = g > 0.0f ? g : 0.0f;
  acc = __fmul_rn(g, g);
  lo = __fadd_rn(jmin.y, sh.y); hi = __fadd_rn(jmax.y, sh.y);
  g1 = __fsub_rn(lo, imax.y); g2 = __fsub_rn(imin.y, hi);
  g = g1 > g2 ? g1 : g2; g = g > 0.0f ? g : 0.0f;
  acc = __fadd_rn(acc, __fmul_rn(g, g));
  lo = __fadd_rn(jmin.z, sh.z); hi = __fadd_rn(jmax.z, sh.z);
  g1 = __fsub_rn(lo, imax.z); g2 = __fsub_rn(imin.z, hi);
  g = g1 > g2 ? g1 : g2; g = g > 0.0f ? g : 0.0f;
  acc = __fadd_rn(acc, __fmul_rn(g, g));
  return acc <= c2;
}

// ---------------------------------------------------------------------------
// 1. Binning: wrap shift, column and z key per atom.
// ---------------------------------------------------------------------------
__global__ void k_bin(Dev d, const float *__restrict__ pos) {
  pdl_wait();
  int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a == 0) atomicAnd(&d.ctr->status, ~kStatusListInvalid);  // this rebuild starts a fresh list
  if (a >= d.N) return;
  const RepInfo &ri = d.rep[d.atomRep[a]];
  const float x = pos[3 * a], y = pos[3 * a + 1], z = pos[3 * a + 2];
  if (!(isfinite(x) && isfinite(y) && isfinite(z))) atomicOr(&d.ctr->status, kStatusNonFinite);
  // Image shift as the reference's triclinic modulus (src/main/real3.h:340-360):
  // z by C, then y by B, then x by A; for an orthorhombic box the three are
  // independent.
  float fz = floorf(__fdiv_rn(z, ri.box[2]));
  fz = fminf(fmaxf(fz, -127.0f), 127.0f);
  const float yz = __fsub_rn(y, __fmul_rn(fz, ri.tric[2]));
  const float xz = __fsub_rn(x, __fmul_rn(fz, ri.tric[1]));
  float fy = floorf(__fdiv_rn(yz, ri.box[1]));
  fy = fminf(fmaxf(fy, -127.0f), 127.0f);
  const float xy = __fsub_rn(xz, __fmul_rn(fy, ri.tric[0]));
  float fx = floorf(__fdiv_rn(xy, ri.box[0]));
  fx = fminf(fmaxf(fx, -127.0f), 127.0f);
  int s[3] = {(int)fx, (int)fy, (int)fz};
  // the packed (wrapped) coordinates, as k_pack computes them
  const float3 L = lattice_shift(ri.box, ri.tric, s[0], s[1], s[2]);
  float w[3] = {__fsub_rn(x, L.x), __fsub_rn(y, L.y), __fsub_rn(z, L.z)};
  d.wrap[a] = (s[0] + 128) | ((s[1] + 128) << 8) | ((s[2] + 128) << 16);
  int ix = (int)floorf(__fmul_rn(__fdiv_rn(w[0], ri.box[0]), (float)ri.divX));
  // far outside the box (more than 127 images): its column's AABB exceeds the column
  bool wide = ix < -1 || ix > ri.divX;
  ix = ix >= ri.divX ? ri.divX - 1 : ix;
  ix = ix < 0 ? 0 : ix;
  int iy = (int)floorf(__fmul_rn(__fdiv_rn(w[1], ri.box[1]), (float)ri.divY));
  wide = wide || iy < -1 || iy > ri.divY;
  if (wide) atomicOr(&d.ctr->wideBin, 1);
  iy = iy >= ri.divY ? ri.divY - 1 : iy;
  iy = iy < 0 ? 0 : iy;
  int col = ri.colStart + ix * ri.divY + iy;
  d.atomCol[a] = col;
  d.atomZKey[a] = z_key(w[2]);
  // place in the column (any order): one atomic for the warp's atoms of a column,
  // which are many, as consecutive atoms are neighbours
  const unsigned peers = __match_any_sync(__activemask(), col);
  const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
  int at = 0;
  if (lane == leader) at = atomicAdd(&d.colCount[col], __popc(peers));
  at = __shfl_sync(peers, at, leader);
  d.atomRank[a] = at + __popc(peers & ((1u << lane) - 1u));
}

// ---------------------------------------------------------------------------
// 2. Column scan (single CTA): atom and block offsets.
// ---------------------------------------------------------------------------
__global__ void k_colscan(Dev d) {
  pdl_wait();
  __shared__ int carryA, carryB;
  if (threadIdx.x == 0) { carryA = 0; carryB = 0; }
  __syncthreads();
  const int nc = d.totalCols;
  for (int c0 = 0; c0 < nc; c0 += blockDim.x) {
    int c = c0 + threadIdx.x;
    int n = c < nc ? d.colCount[c] : 0;
    int nb = (n + 31) >> 5;
    // two block-wide scans via warp shuffles and shared memory
    __shared__ int wa[32], wb[32];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int xa = n, xb = nb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int ya = __shfl_up_sync(kFull, xa, o), yb = __shfl_up_sync(kFull, xb, o);
      if (lane >= o) { xa += ya; xb += yb; }
    }
    if (lane == 31) { wa[w] = xa; wb[w] = xb; }
    __syncthreads();
    if (w == 0) {
      int sa = lane < nw ? wa[lane] : 0, sb = lane < nw ? wb[lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int ya = __shfl_up_sync(kFull, sa, o), yb = __shfl_up_sync(kFull, sb, o);
        if (lane >= o) { sa += ya; sb += yb; }
      }
      if (lane < nw) { wa[lane] = sa; wb[lane] = sb; }
    }
    __syncthreads();
    int offA = carryA + (w ? wa[w - 1] : 0) + xa - n;
    int offB = carryB + (w ? wb[w - 1] : 0) + xb - nb;
    if (c < nc) {
      d.colStartAtom[c] = offA;
      d.colStartBlock[c] = offB;
    }
    __syncthreads();
    if (threadIdx.x == 0) { carryA += wa[nw - 1]; carryB += wb[nw - 1]; }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    int B = carryB;
    d.colStartAtom[nc] = carryA;
    d.colStartBlock[nc] = B;
    if (B > d.maxBlocks) {
      atomicOr(&d.ctr->status, kStatusBlockOverflow);
      B = d.maxBlocks;
    }
    d.blockBounds[B] = carryA;
    d.ctr->blockCount = B;
  }
  if (threadIdx.x == 0) {  // the list of this rebuild is counted afresh
    d.ctr->candCount = d.ctr->maskCount = 0;
    d.ctr->work[0] = d.ctr->work[1] = 0;
    d.ctr->wide = d.ctr->wideBin;
    d.ctr->wideBin = 0;
  }
  if (threadIdx.x == 0) d.ctr->orderValid = 0;  // until the new items are measured
  __syncthreads();
  for (int r = threadIdx.x; r <= d.R; r += blockDim.x) {
    int b = r < d.R ? d.colStartBlock[d.rep[r].colStart] : d.colStartBlock[nc];
    d.repBlockStart[r] = b < d.maxBlocks ? b : d.maxBlocks;
  }
}

// 3. Scatter atoms into column buckets (arbitrary order within a column).
__global__ void k_scatter(Dev d) {
  pdl_wait();
  int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= d.N) return;
  d.bucket[d.colStartAtom[d.atomCol[a]] + d.atomRank[a]] = a;
}

__device__ __forceinline__ float key_float(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k ^ 0x80000000u) : ~k);
}

// Packed position of slot t (atom a of replica ri, -1: empty) into xyzq, and the
// AABBs of its block b and the block's halves; one warp, lane = slot.
__device__ __forceinline__ void pack_slot(const Dev &d, const float *__restrict__ pos, const RepInfo &ri, int t, int b,
                                          int a, float q, float3 &mn, float3 &mx) {
  float3 p = make_float3(1.0e18f, 0.f, 0.f);  // empty slot: outside every cutoff (k_pair)
  mn = make_float3(INFINITY, INFINITY, INFINITY);
  mx = make_float3(-INFINITY, -INFINITY, -INFINITY);
  if (a >= 0) {
    int w = d.wrap[a];
    const float3 L = lattice_shift(ri.box, ri.tric, (w & 0xFF) - 128, ((w >> 8) & 0xFF) - 128,
                                   ((w >> 16) & 0xFF) - 128);
    p.x = __fsub_rn(pos[3 * a], L.x);
    p.y = __fsub_rn(pos[3 * a + 1], L.y);
    p.z = __fsub_rn(pos[3 * a + 2], L.z);
    mn = p;
    mx = p;
  }
  d.xyzq[t] = make_float4(p.x, p.y, p.z, q);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    if (o == 16 && (t & 15) == 0) {  // the halves' own boxes (k_pair)
      d.hmin[t >> 4] = make_float4(mn.x, mn.y, mn.z, 0.f);
      d.hmax[t >> 4] = make_float4(mx.x, mx.y, mx.z, 0.f);
    }
    mn.x = fminf(mn.x, __shfl_xor_sync(kFull, mn.x, o));
    mn.y = fminf(mn.y, __shfl_xor_sync(kFull, mn.y, o));
    mn.z = fminf(mn.z, __shfl_xor_sync(kFull, mn.z, o));
    mx.x = fmaxf(mx.x, __shfl_xor_sync(kFull, mx.x, o));
    mx.y = fmaxf(mx.y, __shfl_xor_sync(kFull, mx.y, o));
    mx.z = fmaxf(mx.z, __shfl_xor_sync(kFull, mx.z, o));
  }
  if ((t & 31) == 0) {
    d.bmin[b] = make_float4(mn.x, mn.y, mn.z, 0.f);
    d.bmax[b] = make_float4(mx.x, mx.y, mx.z, 0.f);
  }
}

// 4. One CTA per column: sort by (z key, atom index), cut into blocks, slots with
//    their per-atom parameters, packed coordinates, block and column AABBs.
//    The sort counts smaller keys up to 512 atoms (one atom a thread, no
//    barriers between steps), is bitonic up to kSortCap, and counts in global
//    memory above.  A block that hits implies its column hits under the rounding
//    of aabb_hit, so the cull may skip columns that miss.
constexpr int kColThreads = 512;
__global__ void __launch_bounds__(kColThreads) k_column(Dev d, const int *__restrict__ colRep,
                                                        const float *__restrict__ pos) {
  pdl_wait();
  __shared__ unsigned long long key[kSortCap];
  __shared__ uint32_t sKey[6];
  const int c = blockIdx.x;
  const int n = d.colCount[c];
  const int base = d.colStartAtom[c];
  if (threadIdx.x < 6) sKey[threadIdx.x] = threadIdx.x < 3 ? 0xFFFFFFFFu : 0u;  // min keys, max keys
  __syncthreads();  // every thread has read the count
  if (n == 0) return;
  if (threadIdx.x == 0) d.colCount[c] = 0;  // zero for the next rebuild's binning
  const bool inShared = n <= kSortCap;
  if (n <= kColThreads) {
    unsigned long long mine = 0;
    const int i = threadIdx.x;
    if (i < n) {
      const int a = d.bucket[base + i];
      mine = ((unsigned long long)d.atomZKey[a] << 32) | (unsigned)a;
      key[i] = mine;
    }
    __syncthreads();
    int rank = 0;
#pragma unroll 8
    for (int j = 0; j < n; j++) rank += key[j] < mine;
    __syncthreads();
    if (i < n) key[rank] = mine;
    __syncthreads();
  } else if (inShared) {
    int n2 = 1;
    while (n2 < n) n2 <<= 1;
    for (int i = threadIdx.x; i < n2; i += blockDim.x) {
      if (i < n) {
        int a = d.bucket[base + i];
        key[i] = ((unsigned long long)d.atomZKey[a] << 32) | (unsigned)a;
      } else {
        key[i] = ~0ull;
      }
    }
    __syncthreads();
    for (int k = 2; k <= n2; k <<= 1) {
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int i = threadIdx.x; i < n2; i += blockDim.x) {
          int ixj = i ^ j;
          if (ixj > i) {
            unsigned long long x = key[i], y = key[ixj];
            bool up = (i & k) == 0;
            if ((x > y) == up) { key[i] = y; key[ixj] = x; }
          }
        }
        __syncthreads();
      }
    }
  } else {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      int a = d.bucket[base + i];
      unsigned long long ki = ((unsigned long long)d.atomZKey[a] << 32) | (unsigned)a;
      int rank = 0;
      for (int j = 0; j < n; j++) {
        int b = d.bucket[base + j];
        unsigned long long kj = ((unsigned long long)d.atomZKey[b] << 32) | (unsigned)b;
        rank += kj < ki;
      }
      d.sortedAtom[base + rank] = a;
    }
    __syncthreads();
  }
  // blocks of 32: one warp each
  const int r = colRep[c];
  const RepInfo &ri = d.rep[r];
  const int b0 = d.colStartBlock[c], nb = (n + 31) >> 5, lane = threadIdx.x & 31;
  for (int k = threadIdx.x >> 5; k < nb; k += kColThreads / 32) {
    const int b = b0 + k, t = 32 * b + lane, i = 32 * k + lane;
    if (b >= d.maxBlocks) break;  // flagged by the column scan
    int a = -1;
    float q = 0.f;
    if (i < n) {
      if (inShared) {
        a = (int)(key[i] & 0xFFFFFFFFull);
        d.sortedAtom[base + i] = a;
      } else {
        a = d.sortedAtom[base + i];
      }
      const int type = d.atomType[a];
      q = d.atomQ[a];
      d.atomSlot[a] = t;
      d.slotQ[t] = q;
      d.slotType[t] = type;
      if (d.ljCombine) d.slotLj[t] = d.ljType[type];
      d.slotSiteBlock[t] = d.atomSiteBlock[a];
    } else {
      d.slotQ[t] = 0.f;
      d.slotType[t] = 0;
      if (d.ljCombine) d.slotLj[t] = make_float2(0.f, 0.f);
      d.slotSiteBlock[t] = 0;
    }
    d.slotAtom[t] = a;
    float3 mn, mx;
    pack_slot(d, pos, ri, t, b, a, q, mn, mx);
    if (lane == 0) {
      d.blockBounds[b] = base + 32 * k;
      d.blockRep[b] = r;
      atomicMin(&sKey[0], z_key(mn.x));
      atomicMin(&sKey[1], z_key(mn.y));
      atomicMin(&sKey[2], z_key(mn.z));
      atomicMax(&sKey[3], z_key(mx.x));
      atomicMax(&sKey[4], z_key(mx.y));
      atomicMax(&sKey[5], z_key(mx.z));
    }
  }
  __syncthreads();
  if (threadIdx.x < 6) d.colKey[6 * c + threadIdx.x] = sKey[threadIdx.x];
}

}  // namespace

// Per step: pack coordinates with the stored image shift; block AABBs.
__global__ void k_pack(Dev d, const float *__restrict__ pos) {
  pdl_wait();
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  int b = t >> 5;
  if (b >= d.maxBlocks) return;
  if (b >= d.ctr->blockCount) return;
  float3 mn, mx;
  pack_slot(d, pos, d.rep[d.blockRep[b]], t, b, d.slotAtom[t], d.slotQ[t], mn, mx);
}

namespace {

// Exclusion word of one atom (lane of iBlock) against the 32 atoms of jBlock: bit
// b is clear where atom b is an excluded partner.
__device__ __forceinline__ uint32_t excl_row(const Dev &d, int iBlock, int jBlock, int lane) {
  uint32_t row = 0xFFFFFFFFu;
  int a = d.slotAtom[32 * iBlock + lane];
  if (a >= 0) {
    int e1 = d.exclStart[a + 1];
    for (int e = d.exclStart[a]; e < e1; e++) {
      int b = d.exclAtom[e];
      if (b == a) continue;
      int sl = d.atomSlot[b];
      if ((sl >> 5) == jBlock) row &= ~(1u << (sl & 31));
    }
  }
  return row;
}

// 5. One CTA per i block.
//    * The blocks that hold an excluded partner of one of its atoms go into a
//      hash table, and their mask words (of j atom l: bit i clear = excluded from
//      i atom i) are made as they are found.  A candidate tile needs a mask
//      exactly if its j block is there; its shift code does not matter.  With more
//      than kPartners distinct blocks every candidate is scanned instead.
//    * Cull: per shift code the j blocks of the replica are visited column by
//      column, over the columns within reach (a column's atoms lie inside it, give
//      or take rounding, unless some atom was out of the box): lanes test the
//      columns' AABBs, the blocks of the columns that hit are concatenated (warp
//      scan of their counts) and tested 32 at a time.  The columns of all codes
//      are cut into at most kTasks pieces for the CTA's warps (most blocks reach
//      no image, so a warp per code would leave one warp all the work).  Columns,
//      and the blocks inside them, are in increasing block order, so the
//      candidates come out in the order of a scan over codes and j blocks.  Hits
//      are kept in shared memory (a piece with more than kHits is visited again).
//    * One atomic each reserves the block's candidates, masks and work items, and
//      the CTA writes them.  Work items: (block and tiles, first candidate), by
//      work_split; the full-size ones from the start of the list, the tail
//      after them (the pair kernel takes items in list order until it has
//      measured them).
//    Bound by the latencies one CTA sees in a row, so by CTAs in flight.  It
//    replaces twelve launches (partner lists, count and write passes of cull and
//    masks with scans between, work list).  Whole rebuild, us, before -> at 4
//    warps a CTA (at 2, 8): 23,558 atoms 117 -> 37 (43, 39), 192,000 atoms
//    557 -> 131 (126, 157), 8 MSLD replicas 200 -> 63 (70, 67), 32 MSLD boxes
//    145 -> 40 (45, 43).
constexpr int kCullWarps = 4, kCullThreads = 32 * kCullWarps;
constexpr int kTasks = 48, kHits = 40, kPartners = 32, kTable = 64, kMaskJobs = 128;

__device__ __forceinline__ unsigned table_slot(int block) { return ((unsigned)block * 0x9E3779B1u) >> 26; }

__global__ void __launch_bounds__(kCullThreads) k_cull(Dev d, float rcull, float rcull2) {
  pdl_wait();
  const int iBlock = blockIdx.x;
  if (iBlock >= d.ctr->blockCount) return;
  __shared__ int sTable[kTable];
  __shared__ uint32_t sWord[kTable][32];
  __shared__ int sPartners;
  __shared__ int sHit[kTasks][kHits];          // j block, sign bit: needs a mask
  __shared__ int sCnt[kTasks], sFlag[kTasks];  // of a piece; later the offsets of its first
  __shared__ int sBase[4];                     // candidates, masks, work items of either part
  __shared__ int sOk, sJobs, sTotal;
  __shared__ int2 sJob[kMaskJobs];             // (j block, mask)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = d.blockRep[iBlock];
  const RepInfo &ri = d.rep[r];
  for (int i = threadIdx.x; i < kTable * 32; i += kCullThreads) (&sWord[0][0])[i] = 0xFFFFFFFFu;
  if (threadIdx.x < kTable) sTable[threadIdx.x] = -1;
  if (threadIdx.x == 0) sPartners = sJobs = 0;
  __syncthreads();
  {
    const int a = d.slotAtom[32 * iBlock + lane];
    const int e0 = a >= 0 ? d.exclStart[a] : 0, e1 = a >= 0 ? d.exclStart[a + 1] : 0;
    for (int e = e0 + warp; e < e1; e += 4 * kCullWarps) {
      int p[4], sl[4];
#pragma unroll
      for (int k = 0; k < 4; k++) p[k] = e + k * kCullWarps < e1 ? d.exclAtom[e + k * kCullWarps] : a;
#pragma unroll
      for (int k = 0; k < 4; k++) sl[k] = d.atomSlot[p[k]];
      for (int k = 0; k < 4; k++) {
        if (p[k] == a || sPartners > kPartners) continue;
        const int jb = sl[k] >> 5;
        unsigned h = table_slot(jb);
        for (int probe = 0; probe < kTable; probe++, h = (h + 1) & (kTable - 1)) {
          const int old = atomicCAS(&sTable[h], -1, jb);
          if (old == -1) atomicAdd(&sPartners, 1);
          if (old == -1 || old == jb) {
            atomicAnd(&sWord[h][sl[k] & 31], ~(1u << lane));
            break;
          }
        }
      }
    }
  }
  const float4 imin = d.bmin[iBlock], imax = d.bmax[iBlock];
  // lane = shift code: columns within reach, one more on each side for rounding
  int x0 = 0, y0 = 0, ny = 0, cells = 0;
  if (lane < kNumShifts) {
    int x1 = ri.divX - 1, y1 = ri.divY - 1;
    if (!d.ctr->wide) {
      const float4 sv = ri.shift[lane];
      const float bx = (float)ri.divX / ri.box[0], by = (float)ri.divY / ri.box[1];
      x0 = max(x0, (int)floorf((imin.x - rcull - sv.x) * bx) - 1);
      x1 = min(x1, (int)floorf((imax.x + rcull - sv.x) * bx) + 1);
      y0 = max(y0, (int)floorf((imin.y - rcull - sv.y) * by) - 1);
      y1 = min(y1, (int)floorf((imax.y + rcull - sv.y) * by) + 1);
    }
    // the box of a block that has no finite x or y is (inf, -inf): its range ends at
    // the limits of int, where a difference would wrap
    if (x0 <= x1 && y0 <= y1) {
      ny = y1 - y0 + 1;
      cells = (x1 - x0 + 1) * ny;
    }
  }
  int all = cells;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) all += __shfl_xor_sync(kFull, all, o);
  const int piece = max(8, (all + 31) / 32);  // columns per piece: at most 32 + kNumShifts pieces
  const int pieces = (cells + piece - 1) / piece;
  int pEnd = pieces;  // lane = code: pieces up to and with this code
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(kFull, pEnd, o);
    if (lane >= o) pEnd += v;
  }
  const int nTasks = __shfl_sync(kFull, pEnd, 31);
  // visit(hit, j, code) for 32 blocks of piece t at a time, in increasing block order
  auto enumerate = [&](int t, auto visit) {
    const int code = __popc(__ballot_sync(kFull, pEnd <= t));
    const int first = (t - (__shfl_sync(kFull, pEnd, code) - __shfl_sync(kFull, pieces, code))) * piece;
    const int cn = __shfl_sync(kFull, cells, code), cx = __shfl_sync(kFull, x0, code);
    const int cy = __shfl_sync(kFull, y0, code), cny = __shfl_sync(kFull, ny, code);
    const int last = min(first + piece, cn);
    const float4 sv = ri.shift[code];
    const float3 sh = make_float3(sv.x, sv.y, sv.z);
    const int j0 = code == 0 ? iBlock : d.repBlockStart[r], j1 = d.repBlockStart[r + 1];
    for (int cb = first; cb < last; cb += 32) {
      int bs = 0, n = 0;
      if (cb + lane < last) {
        const int ix = (cb + lane) / cny, c = ri.colStart + (cx + ix) * ri.divY + cy + (cb + lane - ix * cny);
        bs = d.colStartBlock[c];
        int be = d.colStartBlock[c + 1];
        bs = bs > j0 ? bs : j0;
        be = be < j1 ? be : j1;
        if (bs < be) {
          const uint32_t *key = d.colKey + 6 * c;
          const float4 cmin = make_float4(key_float(key[0]), key_float(key[1]), key_float(key[2]), 0.f);
          const float4 cmax = make_float4(key_float(key[3]), key_float(key[4]), key_float(key[5]), 0.f);
          if (aabb_hit(imin, imax, cmin, cmax, sh, rcull2)) n = be - bs;
        }
      }
      int inc = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, inc, o);
        if (lane >= o) inc += y;
      }
      const int tot = __shfl_sync(kFull, inc, 31);
      const int exc = inc - n;
      for (int t0 = 0; t0 < tot; t0 += 32) {
        const int q = t0 + lane;
        // column lane k holding item q: the first lane whose inclusive count exceeds q
        int k = 0;
#pragma unroll
        for (int step = 16; step > 0; step >>= 1)
          if (__shfl_sync(kFull, inc, k + step - 1) <= q) k += step;
        const int jStart = __shfl_sync(kFull, bs, k);
        const int jOff = __shfl_sync(kFull, exc, k);
        const int j = q < tot ? jStart + (q - jOff) : iBlock;
        visit(q < tot && aabb_hit(imin, imax, d.bmin[j], d.bmax[j], sh, rcull2), j, code);
      }
    }
  };
  __syncthreads();  // the table is complete
  const bool listed = sPartners <= kPartners;
  auto find = [&](int j) {  // slot of block j in the table, -1: not there
    unsigned h = table_slot(j);
    for (int probe = 0; probe < kTable; probe++, h = (h + 1) & (kTable - 1)) {
      const int v = sTable[h];
      if (v == j) return (int)h;
      if (v == -1) break;
    }
    return -1;
  };
  // the lanes' hits that need a mask
  auto masked = [&](bool hit, int j) {
    if (listed) return __ballot_sync(kFull, hit && find(j) >= 0);
    unsigned out = 0;
    for (unsigned m = __ballot_sync(kFull, hit); m; m &= m - 1) {
      const int l = __ffs(m) - 1, jj = __shfl_sync(kFull, j, l);
      if (__any_sync(kFull, excl_row(d, jj, iBlock, lane) != 0xFFFFFFFFu)) out |= 1u << l;
    }
    return out;
  };
  const unsigned before = (1u << lane) - 1u;
  for (int t = warp; t < nTasks; t += kCullWarps) {
    int cnt = 0, flags = 0;
    enumerate(t, [&](bool hit, int j, int) {
      const unsigned m = __ballot_sync(kFull, hit), f = masked(hit, j);
      const int at = cnt + __popc(m & before);
      if (hit && at < kHits) sHit[t][at] = j | ((f >> lane & 1u) ? (int)0x80000000u : 0);
      cnt += __popc(m);
      flags += __popc(f);
    });
    if (lane == 0) {
      sCnt[t] = cnt;
      sFlag[t] = flags;
    }
  }
  __syncthreads();
  __shared__ int sOff[kTasks], sOffF[kTasks];
  if (warp == 0) {  // offsets of the pieces, and the block's place in the list
    int c0 = lane < nTasks ? sCnt[lane] : 0, c1 = 32 + lane < nTasks ? sCnt[32 + lane] : 0;
    int f0 = lane < nTasks ? sFlag[lane] : 0, f1 = 32 + lane < nTasks ? sFlag[32 + lane] : 0;
    auto scan = [&](int v) {
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, v, o);
        if (lane >= o) v += y;
      }
      return v;
    };
    const int i0 = scan(c0), t0 = __shfl_sync(kFull, i0, 31), i1 = scan(c1), total = t0 + __shfl_sync(kFull, i1, 31);
    const int g0 = scan(f0), u0 = __shfl_sync(kFull, g0, 31), g1 = scan(f1), totalF = u0 + __shfl_sync(kFull, g1, 31);
    sOff[lane] = i0 - c0;
    sOffF[lane] = g0 - f0;
    if (32 + lane < kTasks) {
      sOff[32 + lane] = t0 + i1 - c1;
      sOffF[32 + lane] = u0 + g1 - f1;
    }
    int tiles[kWorkLevels], items[kWorkLevels];
    const int L = work_split(total, ri.tilesPerWork, ri.tailTiles, tiles, items);
    int tail = 0;
    for (int l = 1; l < L; l++) tail += items[l];
    int cap = 0, add = 0, *p = nullptr, bit = 0, base = 0;
    if (lane == 0) { p = &d.ctr->candCount; add = total; cap = d.capCand; bit = kStatusCandOverflow; }
    if (lane == 1) { p = &d.ctr->maskCount; add = totalF; cap = d.capMask; bit = kStatusMaskOverflow; }
    if (lane == 2) { p = &d.ctr->work[0]; add = items[0]; cap = d.capWork; bit = kStatusWorkOverflow; }
    if (lane == 3) { p = &d.ctr->work[1]; add = tail; cap = d.capWork; bit = kStatusWorkOverflow; }
    bool fits = true;
    if (lane < 4) {
      base = atomicAdd(p, add);
      fits = base <= cap && add <= cap - base;
      if (!fits) atomicOr(&d.ctr->status, bit);
      sBase[lane] = base;
    }
    const bool ok = __all_sync(kFull, fits);
    if (lane == 0) {
      sOk = ok;
      sTotal = total;
      d.candStart[iBlock] = base;
      d.candNum[iBlock] = ok ? total : 0;
    }
  }
  __syncthreads();
  if (!sOk) return;  // the list is marked invalid: no kernel reads it
  for (int t = warp; t < nTasks; t += kCullWarps) {
    int p = sBase[0] + sOff[t], fm = sBase[1] + sOffF[t];
    const int cnt = sCnt[t];
    auto emit = [&](bool hit, int j, int code, unsigned f) {
      const unsigned m = __ballot_sync(kFull, hit);
      if (hit) {
        int mask = -1;
        if (f >> lane & 1u) {
          mask = fm + __popc(f & before);
          const int job = atomicAdd(&sJobs, 1);
          if (job < kMaskJobs) sJob[job] = make_int2(j, mask);
        }
        d.cand[p + __popc(m & before)] = make_int4(j, code, mask, iBlock);
      }
      p += __popc(m);
      fm += __popc(f);
    };
    if (cnt <= kHits) {
      const int code = __popc(__ballot_sync(kFull, pEnd <= t));
      for (int t0 = 0; t0 < cnt; t0 += 32) {
        const bool hit = t0 + lane < cnt;
        const int v = hit ? sHit[t][t0 + lane] : 0;
        emit(hit, v & 0x7FFFFFFF, code, __ballot_sync(kFull, v < 0));
      }
    } else {
      enumerate(t, [&](bool hit, int j, int code) { emit(hit, j, code, masked(hit, j)); });
    }
  }
  __syncthreads();
  auto word = [&](int j) { return listed ? sWord[find(j) & (kTable - 1)][lane] : excl_row(d, j, iBlock, lane); };
  if (sJobs <= kMaskJobs) {
    for (int k = warp; k < sJobs; k += kCullWarps) d.masks[32 * (size_t)sJob[k].y + lane] = word(sJob[k].x);
  } else {  // more masks than jobs: over the block's candidates (written above)
    for (int k = warp; k < sTotal; k += kCullWarps) {
      const int4 c = d.cand[sBase[0] + k];
      if (c.z >= 0) d.masks[32 * (size_t)c.z + lane] = word(c.x);
    }
  }
  int tiles[kWorkLevels], items[kWorkLevels];
  const int L = work_split(sTotal, ri.tilesPerWork, ri.tailTiles, tiles, items);
  for (int l = 0; l < L; l++) {
    const WorkLevel lv = work_level(sBase[0], ri.tilesPerWork, l, tiles, items);
    int2 *out = (l == 0 ? d.work + sBase[2] : d.work + d.capWork + sBase[3]) + lv.before;
    for (int k = threadIdx.x; k < lv.items; k += kCullThreads) {
      int first, n;
      lv.item(k, &first, &n);
      out[k] = make_int2(work_pack(iBlock, n), first);
    }
  }
}

inline int grid_for(long long n, int threads) {
  long long g = (n + threads - 1) / threads;
  if (g < 1) g = 1;
  if (g > 65535LL * 16) g = 65535LL * 16;
  return (int)g;
}

}  // namespace

void pack_positions(const Dev &d, const float *pos, cudaStream_t s) {
  int n = 32 * d.maxBlocks;
  launch_pdl(k_pack, grid_for(n, 256), 256, 0, s, d, pos);
}

namespace {
__global__ void k_clear_status(Counters *c) {
  pdl_wait();
  atomicAnd(&c->status, ~kStatusListInvalid);
}
}  // namespace

int rebuild_list(const Dev &d, const int *colRep, const float *pos, float rcull, cudaStream_t s) {
  // colCount is zero here: set so at allocation and by k_column after use
  if (d.N > 0) launch_pdl(k_bin, grid_for(d.N, 256), 256, 0, s, d, pos);  // also clears the list-invalid bits
  else launch_pdl(k_clear_status, 1, 1, 0, s, d.ctr);
  launch_pdl(k_colscan, 1, 1024, 0, s, d);
  if (d.N > 0) launch_pdl(k_scatter, grid_for(d.N, 256), 256, 0, s, d);
  launch_pdl(k_column, d.totalCols, kColThreads, 0, s, d, colRep, pos);
  launch_pdl(k_cull, d.maxBlocks, kCullThreads, 0, s, d, rcull, rcull * rcull);
  return d.N > 0 ? 5 : 4;
}

}  // namespace bnb
