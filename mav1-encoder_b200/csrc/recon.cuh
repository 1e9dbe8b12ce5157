// Closed-loop reconstruction (reference src/kernels/k_recon.h,
// scheduled by src/backend_cpu.c:76-156).
//
// Per block in decode order: prediction (inter: 8-tap / compound average /
// optional 3x3 dual-filter search; intra: per transform block from the
// reconstructed neighbours with the spec's BlockDecoded availability),
// forward transform by the Q20 matrices, dead-zone quantisation, eob, and
// the normative inverse transform added back into `rec`; optional luma
// transform-type search and intra tx_depth search by 16 * SSE + lambda * bits.
//
// B200 mapping, per frame:
//  - k_block_map: the unit map, the list of inter blocks, the intra count;
//  - k_recon_inter: persistent 128-thread CTAs take the inter blocks from the
//    list (they read reference pictures only, so none waits);
//  - k_block_deps: each intra block's record and its dependency count (the
//    intra blocks under its edge samples, spec 7.11.2 aboveLimit / leftLimit),
//    its place in those blocks' successor lists; blocks without dependencies
//    seed the ready queue;
//  - k_recon_blocks: the intra blocks as dataflow, luma and chroma as separate
//    tasks with their own persistent workers. Every wait is bounded
//    (Ctx::spin_limit polls); past it the worker sets the error and abort words
//    and every worker stops;
//  - lossless frames: k_recon_lossless, whose blocks do not wait.
// BlockDecoded availability is a function of the decode order (the unit map
// and the corner bits) or of the clear-flags rule (k_recon.h:402-414)
// outside the superblock. Samples of the frame being written are read
// through L2 (ldpx), as other SMs write them during the launch.
#pragma once

#include "common.cuh"
#include "pred.cuh"
#include "tx.cuh"

namespace rec {

// Threads of the CTA coding a block: INTER_THREADS for an inter block,
// INTRA_THREADS for a lossless intra block.
#define RT ((int)blockDim.x)
constexpr int INTER_THREADS = 128, INTRA_THREADS = 128;
#define FWD_SLOT_SIZE 4096
HD int fwd_slot(int kind, int log2n) { return (kind * 5 + log2n - 2) * FWD_SLOT_SIZE; }

// inverse scan tables: position -> scan index, per (scan class, tx size)
__constant__ int d_inv_scan_off[3][19];
__device__ int16_t d_inv_scan[8192];

HD int scan_class(int t) {
  if (t == V_DCT || t == V_ADST || t == V_FLIPADST) return 1;
  if (t == H_DCT || t == H_ADST || t == H_FLIPADST) return 2;
  return 0;
}

struct Ctx {
  const FrameParams *fp;
  const uint8_t *src;
  uint8_t *rec;
  const uint8_t *ref, *gold;
  BlockInfo *blocks;
  const SbInfo *sbs;
  int32_t *coefs;
  const int32_t *mats;
  const int32_t *mats_t;  // the same matrices transposed
  int *status;          // [0] error (1 ready-queue wait, 2 successor list, 4 bulk copy), [1] abort
  const int *blk_at;    // per 4x4 luma unit of the frame: index of the block covering it
  int nblk;             // block slots of the frame
  // the intra blocks' dataflow (below): their records, unfinished
  // dependencies (luma, then chroma), successor lists (blocks whose edges read
  // this block's samples), the ready queues (luma, then chroma; slot value:
  // block index + 1, 0 while the slot is unfilled) and the CNT_ counters
  struct IntraTask *tasks;
  int *dep_count, *succ_count, *succ;
  int *queue, *counters;
  int *inter;           // the inter blocks: large ones from the front, smaller ones from the back
  // polls a dependency wait makes before it gives up (sets the error and
  // abort words); SPIN_LIMIT unless a test shortens it
  int spin_limit;
  // a block index whose luma dependencies are counted once more than they
  // are, so it is never released (-1: none): the failure-detection test's
  // never-released dependency
  int hold;
};

#define MAX_SUCC 96  // successors per block: at most 25 along each edge, with margin
// Ctx::counters: intra blocks, then per kind (luma, chroma) slots claimed, blocks queued, blocks done; the inter blocks of
// at least 32x32 samples, the smaller ones, those taken
enum { CNT_TOTAL, CNT_HEAD, CNT_TAIL = CNT_HEAD + 2, CNT_DONE = CNT_TAIL + 2, CNT_BIG = CNT_DONE + 2, CNT_SMALL, CNT_TAKEN, CNT_WORDS = 16 };

#define TILE_OFF 4     // tile column of the block's first sample (word aligned; the left column at 3)
#define TILE_Y 132     // luma tile stride: TILE_OFF + 2 * 64; rows -1 .. 127
#define TILE_C 68      // chroma tile stride: TILE_OFF + 2 * 32; rows -1 .. 63
#define FMAT_SMALL 336 // 4 * 4 + 8 * 8 + 16 * 16

struct Smem {
  __align__(16) int32_t resid[64 * 64];  // residual, then the inverse transform's plane
  int32_t tmp[64 * 32];    // forward row pass output
  int32_t q[32 * 32];      // levels of the current candidate
  int32_t qbest[32 * 32];  // levels kept by the tx type search
  int sse33[33];
  long long red[8];  // one per warp
  BlockInfo blk;
  int maxLumaW, maxLumaH;
  int flag;
  int r0, c0;  // its superblock's first 4x4 row / column
  // views of the reconstruction and the source: plane origins (absolute
  // plane coordinates) and strides; the frames for an inter block, the
  // tiles below for an intra block
  uint8_t *recp[3];
  int rstride[3];
  const uint8_t *srcp[3];
  int sstride[3];
  FrameParams fpc;           // the CTA's copy of the frame parameters
  uint64_t qinv[3][2];       // per plane: the quantiser's reciprocals of dc_q and ac_q (tx::quant_inv)
  int cornerAR[3], cornerBL[3];  // BlockDecoded of those units
  // What only one of the two kernels uses. k_recon_inter launches with the
  // shared memory up to the end of its part (SMEM_INTER), k_recon_lossless
  // with the whole struct, so neither holds the other's part on its SMs.
  union {
    struct {  // inter blocks
      int16_t pred0[64 * 64];  // first compound prediction (intermediate precision)
      // the superblock's source (luma 64 x 64, then the two 32 x 32 chroma
      // planes), bulk-copied in once per CTA
      __align__(16) uint8_t srcSB[64 * 64 + 2 * 32 * 32];
      // the block plane being coded: prediction, then reconstruction, then
      // written back to the frame
      __align__(16) uint8_t recT[64 * 64];
      __align__(8) unsigned long long bar;  // completion of the source copies
    };
    struct {  // lossless intra blocks
      int edge[3][EDGE_LEN];   // AboveRow, LeftCol, filter copy
      // tiles: rows and columns -1 .. 2n - 1 around the block (its own
      // samples, the above row over the above-right units, the left column
      // over the below-left units), and its source
      uint8_t tileY[TILE_Y * 129];
      uint8_t tileC[2][TILE_C * 65];
      uint8_t srcY[64 * 64];
      uint8_t srcC[2][32 * 32];
    };
  };
};
constexpr size_t SMEM_INTER = offsetof(Smem, bar) + sizeof(unsigned long long);
constexpr size_t SMEM_INTRA = sizeof(Smem);

// Sums / maxima over the CTA.
__device__ __forceinline__ long long cta_sum64(long long v, Smem &sm) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  if ((threadIdx.x & 31) == 0) sm.red[threadIdx.x >> 5] = v;
  __syncthreads();
  long long s = 0;
  for (int k = 0; k < RT / 32; k++) s += sm.red[k];
  __syncthreads();
  return s;
}
__device__ __forceinline__ int cta_max(int v, Smem &sm) {
  for (int off = 16; off > 0; off >>= 1) v = imax(v, __shfl_xor_sync(0xffffffffu, v, off));
  if ((threadIdx.x & 31) == 0) sm.red[threadIdx.x >> 5] = v;
  __syncthreads();
  int m = 0;
  for (int k = 0; k < RT / 32; k++) m = imax(m, (int)sm.red[k]);
  __syncthreads();
  return m;
}

struct CtaSync {
  __device__ void operator()() const { __syncthreads(); }
};

// One row of the inverse transform at a fixed width: dequantised levels ->
// row transform -> clamp, into resid (stride RS).
// RAW: q holds levels, dequantised here; otherwise dequantised levels.
template <int LW, int RS, bool RAW>
__device__ __forceinline__ void inv_row(int32_t *resid, const int32_t *q, int i, int th, int dcQ, int acQ, int denom, int rect, int rk,
                        int rowShift) {
  constexpr int W = 1 << LW, TW = W < 32 ? W : 32;
  int32_t t[W];
  int nz = 0;
#pragma unroll
  for (int j = 0; j < W; j++) {
    int v = (j < TW && i < th) ? q[i * TW + j] : 0;
    t[j] = RAW ? tx::dequant_level(v, (i == 0 && j == 0) ? dcQ : acQ, denom) : v;
    nz |= t[j];
  }
  if (!nz) {
#pragma unroll
    for (int j = 0; j < W; j++) resid[i * RS + j] = 0;
    return;
  }
  if (rect) {
#pragma unroll
    for (int j = 0; j < W; j++) t[j] = (int32_t)round2l((int64_t)t[j] * 2896, 12);
  }
  tx::inverse_1d_n<LW>(t, rk, 16);
#pragma unroll
  for (int j = 0; j < W; j++) resid[i * RS + j] = clip3(-(1 << 15), (1 << 15) - 1, round2(t[j], rowShift));
}

// One column at a fixed height: column transform, then either added into the
// reconstruction (flipped for FLIPADST types) or stored back into resid.
template <int LH, int RS>
__device__ __forceinline__ void inv_col(int32_t *resid, int j, int w, int ck, int fud, int flr, uint8_t *rec, int rs, int x, int y) {
  constexpr int H = 1 << LH;
  int32_t t[H];
#pragma unroll
  for (int i = 0; i < H; i++) t[i] = resid[i * RS + j];
  tx::inverse_1d_n<LH>(t, ck, 16);
  if (rec) {
    uint8_t *col = rec + y * rs + x + (flr ? (w - 1 - j) : j);
#pragma unroll
    for (int i = 0; i < H; i++) {
      uint8_t *o = col + (fud ? (H - 1 - i) : i) * rs;
      *o = (uint8_t)clip1((int)*o + round2(t[i], 4));
    }
  } else {
#pragma unroll
    for (int i = 0; i < H; i++) resid[i * RS + j] = round2(t[i], 4);
  }
}

// The 32- and 64-point DCT rows / columns by two threads each (adjacent
// lanes of one warp; half 0 runs the even half and the first join pairs,
// half 1 the odd half and the rest, tx::idct_odd), which halves the
// sequential butterfly chain of the largest transforms. Each thread loads
// its permuted inputs directly; the pre-join halves meet in resid.
template <int LW, int RS, bool RAW>
__device__ __forceinline__ void inv_row_split(int32_t *resid, const int32_t *q, int i, int half, int th, int dcQ, int acQ, int denom,
                              int rect, int rowShift) {
  constexpr int W = 1 << LW, HW = W / 2, TW = W < 32 ? W : 32;
  unsigned pair = 3u << ((threadIdx.x & 31) & ~1u);
  int32_t t[HW];
  int nz = 0;
#pragma unroll
  for (int k = 0; k < HW; k++) {
    int j = tx::brev(LW, k + half * HW);
    int v = (j < TW && i < th) ? q[i * TW + j] : 0;
    t[k] = RAW ? tx::dequant_level(v, (i == 0 && j == 0) ? dcQ : acQ, denom) : v;
    nz |= t[k];
  }
  nz |= __shfl_xor_sync(pair, nz, 1);
  int32_t *row = resid + i * RS;
  if (!nz) {
#pragma unroll
    for (int k = 0; k < HW; k++) row[k + half * HW] = 0;
    return;
  }
  if (rect) {
#pragma unroll
    for (int k = 0; k < HW; k++) t[k] = (int32_t)round2l((int64_t)t[k] * 2896, 12);
  }
  if (half == 0) tx::idct<LW - 1, false>(t, 16);
  else tx::idct_odd<LW>(t, 16);
#pragma unroll
  for (int k = 0; k < HW; k++) row[k + half * HW] = t[k];
  __syncwarp(pair);
#pragma unroll
  for (int k = 0; k < HW / 2; k++) {
    int a = k + half * (HW / 2), b = W - 1 - a;
    int32_t va = row[a], vb = row[b];
    tx::idct_join_pair(&va, &vb, 16);
    row[a] = clip3(-(1 << 15), (1 << 15) - 1, round2(va, rowShift));
    row[b] = clip3(-(1 << 15), (1 << 15) - 1, round2(vb, rowShift));
  }
}

template <int LH, int RS>
__device__ __forceinline__ void inv_col_split(int32_t *resid, int j, int half, int w, int fud, int flr, uint8_t *rec, int rs, int x, int y) {
  constexpr int H = 1 << LH, HH = H / 2;
  unsigned pair = 3u << ((threadIdx.x & 31) & ~1u);
  int32_t t[HH];
#pragma unroll
  for (int k = 0; k < HH; k++) t[k] = resid[tx::brev(LH, k + half * HH) * RS + j];
  __syncwarp(pair);  // both halves read before the column is overwritten
  if (half == 0) tx::idct<LH - 1, false>(t, 16);
  else tx::idct_odd<LH>(t, 16);
#pragma unroll
  for (int k = 0; k < HH; k++) resid[(k + half * HH) * RS + j] = t[k];
  __syncwarp(pair);
  uint8_t *col = rec ? rec + y * rs + x + (flr ? (w - 1 - j) : j) : nullptr;
#pragma unroll
  for (int k = 0; k < HH / 2; k++) {
    int a = k + half * (HH / 2), b = H - 1 - a;
    int32_t va = resid[a * RS + j], vb = resid[b * RS + j];
    tx::idct_join_pair(&va, &vb, 16);
    if (rec) {
      uint8_t *oa = col + (fud ? (H - 1 - a) : a) * rs, *ob = col + (fud ? (H - 1 - b) : b) * rs;
      *oa = (uint8_t)clip1((int)*oa + round2(va, 4));
      *ob = (uint8_t)clip1((int)*ob + round2(vb, 4));
    } else {
      resid[a * RS + j] = round2(va, 4);
      resid[b * RS + j] = round2(vb, 4);
    }
  }
}

// Levels of a candidate -> reconstruction residual (spec 7.13.3 with the
// dequantisation of 7.12.3), into sm.resid (stride 64).
// With rec set, the column pass adds its output straight into the
// reconstruction (flipped for FLIPADST types) instead of storing it. Every
// length is in it, so it is out of line: the kernel keeps its register budget,
// and the 32- and 64-point passes spill here (1,072 bytes a thread).
__device__ __noinline__ void inverse_2d_any(Smem &sm, const int32_t *q, int txSz, int txType, int dcQ, int acQ,
                                            uint8_t *rec, int rs, int x, int y) {
  int lw = T(Tx_Width_Log2)[txSz], lh = T(Tx_Height_Log2)[txSz];
  int w = 1 << lw, h = 1 << lh, th = imin(32, h);
  int rowShift = T(Transform_Row_Shift)[txSz], denom = tx::dq_denom(txSz);
  int rect = iabs(lw - lh) == 1;
  int rk = tx::row_kind(txType), ck = tx::col_kind(txType);
  if (lw >= 5 && rk == tx::KIND_DCT) {
    for (int p = threadIdx.x; p < 2 * h; p += RT) {
      if (lw == 5) inv_row_split<5, 64, true>(sm.resid, q, p >> 1, p & 1, th, dcQ, acQ, denom, rect, rowShift);
      else inv_row_split<6, 64, true>(sm.resid, q, p >> 1, p & 1, th, dcQ, acQ, denom, rect, rowShift);
    }
  } else for (int i = threadIdx.x; i < h; i += RT) {
    switch (lw) {
      case 2: inv_row<2, 64, true>(sm.resid, q, i, th, dcQ, acQ, denom, rect, rk, rowShift); break;
      case 3: inv_row<3, 64, true>(sm.resid, q, i, th, dcQ, acQ, denom, rect, rk, rowShift); break;
      case 4: inv_row<4, 64, true>(sm.resid, q, i, th, dcQ, acQ, denom, rect, rk, rowShift); break;
      case 5: inv_row<5, 64, true>(sm.resid, q, i, th, dcQ, acQ, denom, rect, rk, rowShift); break;
      default: inv_row<6, 64, true>(sm.resid, q, i, th, dcQ, acQ, denom, rect, rk, rowShift); break;
    }
  }
  __syncthreads();
  int fud = tx::flip_ud(txType), flr = tx::flip_lr(txType);
  if (lh >= 5 && ck == tx::KIND_DCT) {
    for (int p = threadIdx.x; p < 2 * w; p += RT) {
      if (lh == 5) inv_col_split<5, 64>(sm.resid, p >> 1, p & 1, w, fud, flr, rec, rs, x, y);
      else inv_col_split<6, 64>(sm.resid, p >> 1, p & 1, w, fud, flr, rec, rs, x, y);
    }
  } else for (int j = threadIdx.x; j < w; j += RT) {
    switch (lh) {
      case 2: inv_col<2, 64>(sm.resid, j, w, ck, fud, flr, rec, rs, x, y); break;
      case 3: inv_col<3, 64>(sm.resid, j, w, ck, fud, flr, rec, rs, x, y); break;
      case 4: inv_col<4, 64>(sm.resid, j, w, ck, fud, flr, rec, rs, x, y); break;
      case 5: inv_col<5, 64>(sm.resid, j, w, ck, fud, flr, rec, rs, x, y); break;
      default: inv_col<6, 64>(sm.resid, j, w, ck, fud, flr, rec, rs, x, y); break;
    }
  }
  __syncthreads();
}

__device__ __forceinline__ void inverse_2d(Smem &sm, const int32_t *q, int txSz, int txType, int dcQ, int acQ,
                                           uint8_t *rec = nullptr, int rs = 0, int x = 0, int y = 0) {
  if (threadIdx.x == 0) {  // h rows of w points, then w columns of h points: 3 log2 N operations per point
    int lw = T(Tx_Width_Log2)[txSz], lh = T(Tx_Height_Log2)[txSz];
    WORK(W_REC_INV_OPS, 3 * (1 << (lw + lh)) * (lw + lh));
  }
  inverse_2d_any(sm, q, txSz, txType, dcQ, acQ, rec, rs, x, y);
}

// The transpose of every forward matrix (slot k: kind k / 5, length 4 << k % 5).
__global__ void k_transpose_mats(const int32_t *mats, int32_t *matsT) {
  int slot = blockIdx.x, n = 4 << (slot % 5);
  const int32_t *m = mats + slot * FWD_SLOT_SIZE;
  int32_t *t = matsT + slot * FWD_SLOT_SIZE;
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) t[(e % n) * n + e / n] = m[e];
}

// Forward row pass: rows of the residual (RS apart) times the kept 32 (or w)
// rows of the Q20 matrix (read from its transpose MhT), 64-bit sums rounded by
// 16 bits into tmp (32 apart), by nt threads. Lengths up to 16: a thread an
// output. Lengths 32 and 64: a warp takes 4 rows, a lane an output column, so
// 4 matrix words and 4 16-byte residual words (the same for the whole warp)
// serve 16 products; an output a thread, two loads a product, left the
// multipliers waiting for shared memory.
template <int LW, int RS>
__device__ __forceinline__ void fwd_rows(const int32_t *resid, int32_t *tmp, const int32_t *MhT, int h, int tid, int nt) {
  constexpr int W = 1 << LW;
  if constexpr (LW <= 4) {
    for (int k = tid; k < h << LW; k += nt) {
      int i = k >> LW, kk = k & (W - 1);
      const int32_t *r = resid + i * RS, *m = MhT + kk;
      int64_t s = 0;
#pragma unroll
      for (int j = 0; j < W; j++) s += (int64_t)r[j] * m[j * W];
      tmp[i * 32 + kk] = (int32_t)round2l(s, 16);
    }
  } else {
    static_assert(RS % 4 == 0, "16-byte residual words");
    const int kk = tid & 31;
    for (int i = (tid >> 5) * 4; i < h; i += nt >> 3) {
      int64_t s[4] = {0, 0, 0, 0};
#pragma unroll 4
      for (int j = 0; j < W; j += 4) {
        int32_t m[4];
#pragma unroll
        for (int q = 0; q < 4; q++) m[q] = MhT[(j + q) * W + kk];
#pragma unroll
        for (int r = 0; r < 4; r++) {
          int4 v = *(const int4 *)(resid + (i + r) * RS + j);
          s[r] += (int64_t)v.x * m[0];
          s[r] += (int64_t)v.y * m[1];
          s[r] += (int64_t)v.z * m[2];
          s[r] += (int64_t)v.w * m[3];
        }
      }
#pragma unroll
      for (int r = 0; r < 4; r++) tmp[(i + r) * 32 + kk] = (int32_t)round2l(s[r], 16);
    }
  }
}
template <int RS>
__device__ __forceinline__ void fwd_rows_any(int lw, const int32_t *resid, int32_t *tmp, const int32_t *MhT, int h, int tid, int nt) {
  switch (lw) {
    case 2: fwd_rows<2, RS>(resid, tmp, MhT, h, tid, nt); break;
    case 3: fwd_rows<3, RS>(resid, tmp, MhT, h, tid, nt); break;
    case 4: fwd_rows<4, RS>(resid, tmp, MhT, h, tid, nt); break;
    case 5: fwd_rows<5, RS>(resid, tmp, MhT, h, tid, nt); break;
    default: if (RS > 64 || RS == 64) fwd_rows<6, RS>(resid, tmp, MhT, h, tid, nt); break;
  }
}

// Forward column pass: emit(k, sum) for output k = k2 * tw + kk of the th x tw
// kept ones. The same split: lengths 32 and 64 give a thread 4 outputs of a
// column.
template <int LH, class Emit>
__device__ __forceinline__ void fwd_cols(const int32_t *tmp, const int32_t *Mv, int ltw, int tid, int nt, Emit emit) {
  constexpr int H = 1 << LH, TH = H < 32 ? H : 32;
  const int tw = 1 << ltw, kk = tid & (tw - 1);  // nt is a multiple of tw
  if constexpr (LH <= 4) {
    for (int k = tid; k < TH << ltw; k += nt) {
      const int32_t *m = Mv + (k >> ltw) * H;
      int64_t s = 0;
#pragma unroll
      for (int i = 0; i < H; i++) s += (int64_t)m[i] * tmp[i * 32 + kk];
      emit(k, s);
    }
  } else {
    for (int k2 = (tid >> ltw) * 4; k2 < TH; k2 += (nt >> ltw) * 4) {
      int64_t s[4] = {0, 0, 0, 0};
#pragma unroll 4
      for (int i = 0; i < H; i += 4) {
        int32_t v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) v[q] = tmp[(i + q) * 32 + kk];
#pragma unroll
        for (int r = 0; r < 4; r++) {
          int4 m = *(const int4 *)(Mv + (k2 + r) * H + i);
          s[r] += (int64_t)m.x * v[0];
          s[r] += (int64_t)m.y * v[1];
          s[r] += (int64_t)m.z * v[2];
          s[r] += (int64_t)m.w * v[3];
        }
      }
#pragma unroll
      for (int r = 0; r < 4; r++) emit((k2 + r) << ltw | kk, s[r]);
    }
  }
}
template <class Emit>
__device__ __forceinline__ void fwd_cols_any(int lh, const int32_t *tmp, const int32_t *Mv, int ltw, int tid, int nt, Emit emit) {
  switch (lh) {
    case 2: fwd_cols<2>(tmp, Mv, ltw, tid, nt, emit); break;
    case 3: fwd_cols<3>(tmp, Mv, ltw, tid, nt, emit); break;
    case 4: fwd_cols<4>(tmp, Mv, ltw, tid, nt, emit); break;
    case 5: fwd_cols<5>(tmp, Mv, ltw, tid, nt, emit); break;
    default: fwd_cols<6>(tmp, Mv, ltw, tid, nt, emit); break;
  }
}
// A column sum as the quantiser takes it (k_fwd.h:92-110).
__device__ __forceinline__ int fwd_scale(int64_t s, int shifts, int rect) {
  s = s * ((int64_t)1 << shifts);
  if (rect) s = round2l(s, 12) * 5793;
  return (int)(s >= 0 ? round2l(s, 20) : -round2l(-s, 20));
}

// ---- one transform type candidate in a warp -------------------------------------------
// Scratch: residual, then the inverse transform (rows CAND_RS apart), the
// forward row pass, the levels.
constexpr int CAND_RS = 17;
struct Cand {
  int32_t r[16 * CAND_RS], t[16 * CAND_RS], q[256];
};
// Source and prediction at the transform block, the forward matrices (rows
// transposed), the quantiser's steps and reciprocals, lambda.
struct CandIn {
  const uint8_t *sp, *pp;
  int ss, ps;
  const int32_t *Mh, *Mv;
  int dcQ, acQ;
  uint64_t invDc, invAc;
  int lambda;
};
template <int LW>
__device__ __forceinline__ void cand_rows(Cand &cd, const int32_t *MhT, int h, int lane) {
  constexpr int W = 1 << LW;
  for (int k = lane; k < h << LW; k += 32) {
    int i = k >> LW, kk = k & (W - 1);
    const int32_t *r = cd.r + i * CAND_RS, *m = MhT + kk;
    int64_t s = 0;
#pragma unroll
    for (int j = 0; j < W; j++) s += (int64_t)r[j] * m[j * W];
    cd.t[i * CAND_RS + kk] = (int32_t)round2l(s, 16);
  }
}
template <int LH>
__device__ __forceinline__ int64_t cand_col(const Cand &cd, const int32_t *Mv, int k2, int kk) {
  constexpr int H = 1 << LH;
  const int32_t *m = Mv + k2 * H;
  int64_t s = 0;
#pragma unroll
  for (int i = 0; i < H; i++) s += (int64_t)m[i] * cd.t[i * CAND_RS + kk];
  return s;
}
__device__ __forceinline__ int level_bits(int l) { return l == 0 ? 6 : 8 * (2 + 2 * (31 - __clz(iabs(l)))); }

// One candidate type of a transform block up to 16 x 16 by one warp (the
// candidate loop of code_tx_block, k_recon.h:101-153): its levels in cd.q, its
// residual in cd.r (flipped types: in transform order), its eob; returns its
// cost.
__device__ __noinline__ long long cand_cost(const CandIn &in, Cand &cd, int type, int txSz, int lane, int *eobOut) {
  const int lw = T(Tx_Width_Log2)[txSz], lh = T(Tx_Height_Log2)[txSz], w = 1 << lw, h = 1 << lh, n = 1 << (lw + lh);
  const int fx = tx::flip_lr(type) ? w - 1 : 0, fy = tx::flip_ud(type) ? h - 1 : 0;  // j ^ fx mirrors j
  for (int k = lane; k < n; k += 32) {
    int i = k >> lw, j = k & (w - 1), y = i ^ fy, x = j ^ fx;
    cd.r[i * CAND_RS + j] = (int)in.sp[y * in.ss + x] - (int)in.pp[y * in.ps + x];
  }
  __syncwarp();
  const int rk = tx::row_kind(type), ck = tx::col_kind(type);
  if (lane == 0) {
    WORK(W_REC_FWD_MAC, n * w + n * h);
    WORK(W_REC_QUANT, n);
  }
  if (lw == 2) cand_rows<2>(cd, in.Mh, h, lane);
  else if (lw == 3) cand_rows<3>(cd, in.Mh, h, lane);
  else cand_rows<4>(cd, in.Mh, h, lane);
  __syncwarp();
  const int shifts = T(Transform_Row_Shift)[txSz] + 4, rect = iabs(lw - lh) == 1;
  const int16_t *inv = d_inv_scan + d_inv_scan_off[scan_class(type)][txSz];
  int eob = 0;
  for (int k = lane; k < n; k += 32) {
    int k2 = k >> lw, kk = k & (w - 1);
    int64_t s = lh == 2 ? cand_col<2>(cd, in.Mv, k2, kk) : lh == 3 ? cand_col<3>(cd, in.Mv, k2, kk) : cand_col<4>(cd, in.Mv, k2, kk);
    int first = k == 0;
    int lv = tx::quant_level(fwd_scale(s, shifts, rect), first ? in.dcQ : in.acQ, first ? 26 : 22, 1, first ? in.invDc : in.invAc);  // dq_denom 1 up to 16 x 16
    cd.q[k] = lv;
    if (lv) eob = imax(eob, inv[k] + 1);
  }
  eob = __reduce_max_sync(0xffffffffu, eob);
  __syncwarp();
  int bits = 0, sse = 0;
  if (eob == 0) {
    bits = 8;
    for (int k = lane; k < n; k += 32) {
      int d = cd.r[(k >> lw) * CAND_RS + (k & (w - 1))];
      sse += d * d;
    }
  } else {
    for (int k = lane; k < n; k += 32)
      if (inv[k] < eob) bits += level_bits(cd.q[k]);
    bits = __reduce_add_sync(0xffffffffu, bits) + 8 * 6 + 8 * 2 * (31 - __clz(eob + 1));
    const int rowShift = T(Transform_Row_Shift)[txSz];
    if (lane == 0) WORK(W_REC_INV_OPS, 3 * n * (lw + lh));
    if (lane < h) {
      if (lw == 2) inv_row<2, CAND_RS, true>(cd.r, cd.q, lane, h, in.dcQ, in.acQ, 1, rect, rk, rowShift);
      else if (lw == 3) inv_row<3, CAND_RS, true>(cd.r, cd.q, lane, h, in.dcQ, in.acQ, 1, rect, rk, rowShift);
      else inv_row<4, CAND_RS, true>(cd.r, cd.q, lane, h, in.dcQ, in.acQ, 1, rect, rk, rowShift);
    }
    __syncwarp();
    if (lane < w) {
      if (lh == 2) inv_col<2, CAND_RS>(cd.r, lane, w, ck, 0, 0, nullptr, 0, 0, 0);
      else if (lh == 3) inv_col<3, CAND_RS>(cd.r, lane, w, ck, 0, 0, nullptr, 0, 0, 0);
      else inv_col<4, CAND_RS>(cd.r, lane, w, ck, 0, 0, nullptr, 0, 0, 0);
    }
    __syncwarp();
    for (int k = lane; k < n; k += 32) {
      int i = k >> lw, j = k & (w - 1), y = i ^ fy, x = j ^ fx;
      int d = (int)in.sp[y * in.ss + x] - clip1((int)in.pp[y * in.ps + x] + cd.r[i * CAND_RS + j]);
      sse += d * d;
    }
  }
  sse = __reduce_add_sync(0xffffffffu, sse);  // at most 256 * 255^2
  *eobOut = eob;
  return (long long)sse * 16 + (long long)in.lambda * bits / 8;
}

// The type search of an inter transform block up to 16 x 16 (up to 16
// candidates): the CTA's warps take them in turn, each keeping its best one's
// scratch, and the first least cost is written out. Returns the eob.
__device__ __noinline__ int search_types(const Ctx &c, Smem &sm, const uint8_t *sp, int ss, uint8_t *pp, int ps, int txSz, int plane,
                                         const int *cands, int numCands, int32_t *coefOut, int *outType) {
  const FrameParams *fp = c.fp;
  constexpr int WARPS = INTER_THREADS / 32;
  static_assert(2 * WARPS * sizeof(Cand) <= offsetof(Smem, sse33), "two candidates a warp in the transform scratch");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lw = T(Tx_Width_Log2)[txSz], lh = T(Tx_Height_Log2)[txSz], w = 1 << lw, h = 1 << lh;
  Cand *own = (Cand *)sm.resid + 2 * warp;
  long long best = -1;
  int bestI = 16, bestEob = 0, bestBuf = 0, cur = 0;
  __syncthreads();
  for (int ci = warp; ci < numCands; ci += WARPS) {
    const int t = cands[ci];
    const CandIn in = {sp, pp, ss, ps, c.mats_t + fwd_slot(tx::row_kind(t), lw), c.mats + fwd_slot(tx::col_kind(t), lh),
                       fp->dc_q[plane], fp->ac_q[plane], sm.qinv[plane][0], sm.qinv[plane][1], fp->lambda};
    int eob;
    long long cost = cand_cost(in, own[cur], t, txSz, lane, &eob);
    if (best < 0 || cost < best) {
      best = cost;
      bestI = ci;
      bestEob = eob;
      bestBuf = cur;
      cur ^= 1;
    }
  }
  if (lane == 0) {
    sm.red[warp] = best;
    sm.sse33[warp] = bestI;
    sm.sse33[8 + warp] = bestEob;
    sm.sse33[16 + warp] = bestBuf;
  }
  __syncthreads();
  int bw = 0;
  best = sm.red[0];
  for (int k = 1; k < WARPS; k++)
    if (sm.red[k] >= 0 && (sm.red[k] < best || (sm.red[k] == best && sm.sse33[k] < sm.sse33[bw]))) {
      best = sm.red[k];
      bw = k;
    }
  const int type = cands[sm.sse33[bw]], eob = sm.sse33[8 + bw];
  const Cand &cd = ((Cand *)sm.resid)[2 * bw + sm.sse33[16 + bw]];
  const int fx = tx::flip_lr(type) ? w - 1 : 0, fy = tx::flip_ud(type) ? h - 1 : 0;
  for (int k = threadIdx.x; k < w * h; k += RT) {
    coefOut[k] = cd.q[k];
    if (eob) {
      int i = k >> lw, j = k & (w - 1);
      uint8_t *o = pp + (i ^ fy) * ps + (j ^ fx);
      *o = (uint8_t)clip1((int)*o + cd.r[i * CAND_RS + j]);
    }
  }
  __syncthreads();
  *outType = eob ? type : DCT_DCT;
  return eob;
}

// A lossless 4x4 transform block whose prediction is in `rec`: transform,
// levels and reconstruction by one thread. Returns the eob.
__device__ int code_wht(const Ctx &c, Smem &sm, const uint8_t *src, int stride, uint8_t *rec, int rs, int x, int y, int plane,
                        int32_t *coefOut) {
  const int dcQ = c.fp->dc_q[plane], acQ = c.fp->ac_q[plane], tid = threadIdx.x;
  // 4x4 Walsh-Hadamard, exact inverse of the spec's (k_fwd.h:112-136); one thread
  if (tid == 0) {
    int r[16], t[16];
    for (int i = 0; i < 4; i++)
      for (int j = 0; j < 4; j++) r[i * 4 + j] = (int)src[(y + i) * stride + x + j] - (int)rec[(y + i) * rs + x + j];
    for (int j = 0; j < 4; j++) {
      int a1 = r[0 * 4 + j], b1 = r[1 * 4 + j], c1 = r[2 * 4 + j], d1 = r[3 * 4 + j];
      a1 += b1;
      d1 = d1 - c1;
      int e1 = (a1 - d1) >> 1;
      b1 = e1 - b1;
      c1 = e1 - c1;
      a1 -= c1;
      d1 += b1;
      t[0 * 4 + j] = a1; t[1 * 4 + j] = c1; t[2 * 4 + j] = d1; t[3 * 4 + j] = b1;
    }
    for (int i = 0; i < 4; i++) {
      int a1 = t[i * 4 + 0], b1 = t[i * 4 + 1], c1 = t[i * 4 + 2], d1 = t[i * 4 + 3];
      a1 += b1;
      d1 -= c1;
      int e1 = (a1 - d1) >> 1;
      b1 = e1 - b1;
      c1 = e1 - c1;
      a1 -= c1;
      d1 += b1;
      sm.q[i * 4 + 0] = a1; sm.q[i * 4 + 1] = c1; sm.q[i * 4 + 2] = d1; sm.q[i * 4 + 3] = b1;
    }
    int eob = 0;
    const int16_t *inv = d_inv_scan + d_inv_scan_off[0][TX_4X4];
    for (int k = 0; k < 16; k++) {
      coefOut[k] = sm.q[k];
      if (sm.q[k] != 0) eob = imax(eob, inv[k] + 1);
    }
    if (eob > 0) {
      int32_t rr[4][4];
      for (int i = 0; i < 4; i++) {
        int32_t tt[4];
        for (int j = 0; j < 4; j++) tt[j] = tx::dequant_level(sm.q[i * 4 + j], (i == 0 && j == 0) ? dcQ : acQ, 1);
        tx::iwht(tt, 2);
        for (int j = 0; j < 4; j++) rr[i][j] = tt[j];
      }
      for (int j = 0; j < 4; j++) {
        int32_t tt[4];
        for (int i = 0; i < 4; i++) tt[i] = clip3(-(1 << 15), (1 << 15) - 1, rr[i][j]);
        tx::iwht(tt, 0);
        for (int i = 0; i < 4; i++) rr[i][j] = tt[i];
      }
      for (int i = 0; i < 4; i++)
        for (int j = 0; j < 4; j++) {
          int o = (y + i) * rs + x + j;
          rec[o] = (uint8_t)clip1((int)rec[o] + rr[i][j]);
        }
    }
    sm.flag = eob;
  }
  __syncthreads();
  int eob = sm.flag;
  __syncthreads();
  return eob;
}

// Transform, quantise and reconstruct one inter transform block whose prediction
// is in `rec` (code_tx_block, k_recon.h:60-173). Returns the eob.
__device__ __forceinline__ int code_tx(const Ctx &c, Smem &sm, const uint8_t *src, int stride, uint8_t *rec, int rs, int x, int y, int txSz,
                       int plane, const int *cands, int numCands, int32_t *coefOut, int *outType) {
  const FrameParams *fp = c.fp;
  int lw = T(Tx_Width_Log2)[txSz], lh = T(Tx_Height_Log2)[txSz];
  int w = 1 << lw, h = 1 << lh, tw = imin(32, w), th = imin(32, h);
  int dcQ = fp->dc_q[plane], acQ = fp->ac_q[plane];
  int tid = threadIdx.x;
  if (numCands > 1 && lw <= 4 && lh <= 4)
    return search_types(c, sm, src + y * stride + x, stride, rec + y * rs + x, rs, txSz, plane, cands, numCands, coefOut, outType);
  // an inter block has no depth search: a single candidate needs no cost
  int single = numCands == 1;
  int shifts = T(Transform_Row_Shift)[txSz] + 4, rect = iabs(lw - lh) == 1;
  int denom = tx::dq_denom(txSz);
  uint64_t invDc = sm.qinv[plane][0], invAc = sm.qinv[plane][1];  // derived once per CTA (load_shared)
  long long bestCost = -1;
  int bestType = DCT_DCT, bestEob = 0;
  int32_t *qsrc = sm.q;  // levels the final reconstruction uses
  for (int ci = 0; ci < numCands; ci++) {
    int t = cands[ci];
    int fud = tx::flip_ud(t), flr = tx::flip_lr(t);
    for (int k = tid; k < h * w; k += RT) {
      int i = k >> lw, j = k & (w - 1);
      int yy = fud ? (h - 1 - i) : i, xx = flr ? (w - 1 - j) : j;
      sm.resid[i * 64 + j] = (int)src[(y + yy) * stride + x + xx] - (int)rec[(y + yy) * rs + x + xx];
    }
    __syncthreads();
    const int32_t *Mh = c.mats_t + fwd_slot(tx::row_kind(t), lw), *Mv = c.mats + fwd_slot(tx::col_kind(t), lh);
    if (tid == 0) {  // row pass h x tw outputs of w terms, column pass th x tw outputs of h terms
      WORK(W_REC_FWD_MAC, h * tw * w + th * tw * h);
      WORK(W_REC_QUANT, th * tw);
    }
    fwd_rows_any<64>(lw, sm.resid, sm.tmp, Mh, h, tid, RT);
    __syncthreads();
    const int16_t *inv = d_inv_scan + d_inv_scan_off[scan_class(t)][txSz];
    int myEob = 0, myNz = 0;
    int ltw = imin(5, lw);
    fwd_cols_any(lh, sm.tmp, Mv, ltw, tid, RT, [&](int k, int64_t s) {
      int first = k == 0;
      int lv = tx::quant_level(fwd_scale(s, shifts, rect), first ? dcQ : acQ, first ? 26 : 22, denom, first ? invDc : invAc);
      sm.q[k] = lv;
      myNz |= lv != 0;
      if (!single && lv != 0) myEob = imax(myEob, inv[k] + 1);
    });
    if (single) {
      // only "has coefficients" matters here (the writer derives the eob)
      int nz = __syncthreads_or(myNz);
      for (int k = tid; k < tw * th; k += RT) coefOut[k] = sm.q[k];
      if (nz) inverse_2d(sm, sm.q, txSz, t, dcQ, acQ, rec, rs, x, y);
      *outType = nz ? t : DCT_DCT;
      return nz;
    }
    int eob = cta_max(myEob, sm);  // includes the barrier after the quantiser
    long long sse = 0;
    if (eob > 0) {
      // keep the residual-free path's SSE source intact: the inverse reuses resid
      inverse_2d(sm, sm.q, txSz, t, dcQ, acQ);
      for (int k = tid; k < h * w; k += RT) {
        int i = k >> lw, j = k & (w - 1);
        int yy = fud ? (h - 1 - i) : i, xx = flr ? (w - 1 - j) : j;
        int d = (int)src[(y + yy) * stride + x + xx] - clip1((int)rec[(y + yy) * rs + x + xx] + sm.resid[i * 64 + j]);
        sse += d * d;
      }
    } else {
      for (int k = tid; k < h * w; k += RT) {
        int i = k >> lw, j = k & (w - 1);
        int d = sm.resid[i * 64 + j];
        sse += d * d;
      }
    }
    sse = cta_sum64(sse, sm);
    long long bits = 0;
    if (eob == 0) {
      bits = tid == 0 ? 8 : 0;
    } else {
      for (int k = tid; k < th * tw; k += RT)
        if (inv[k] < eob) {
          int l = iabs(sm.q[k]);
          bits += l == 0 ? 6 : 8 * (2 + 2 * floor_log2(l));
        }
      if (tid == 0) bits += 8 * 6 + 8 * 2 * floor_log2(eob + 1);
    }
    bits = cta_sum64(bits, sm);
    long long cost = sse * 16 + (long long)fp->lambda * bits / 8;
    if (bestCost < 0 || cost < bestCost) {
      bestCost = cost;
      bestType = eob > 0 ? t : DCT_DCT;
      bestEob = eob;
      for (int k = tid; k < tw * th; k += RT) sm.qbest[k] = sm.q[k];
      qsrc = sm.qbest;
      __syncthreads();
    }
  }
  for (int k = tid; k < tw * th; k += RT) coefOut[k] = qsrc[k];
  if (bestEob > 0) {
    int fud = tx::flip_ud(bestType), flr = tx::flip_lr(bestType);
    if (numCands > 1) inverse_2d(sm, qsrc, txSz, bestType, dcQ, acQ);
    for (int k = tid; k < h * w; k += RT) {
      int i = k >> lw, j = k & (w - 1);
      int yy = fud ? (h - 1 - i) : i, xx = flr ? (w - 1 - j) : j;
      int o = (y + yy) * rs + x + xx;
      rec[o] = (uint8_t)clip1((int)rec[o] + sm.resid[i * 64 + j]);
    }
  }
  __syncthreads();
  *outType = bestType;
  return bestEob;
}

__device__ __forceinline__ void tx_type_set(BlockInfo &b, int idx, int t) {
  if (idx >= 16) return;
  int sh = 4 * (idx & 7);
  if (idx < 8) b.tx_types_lo = (int32_t)(((uint32_t)b.tx_types_lo & ~(15u << sh)) | ((uint32_t)t << sh));
  else b.tx_types_hi = (int32_t)(((uint32_t)b.tx_types_hi & ~(15u << sh)) | ((uint32_t)t << sh));
}

// CfL alpha of one chroma transform block: first minimum of the SSE over
// alpha in [-16, 16] (cfl_best_alpha, k_intra.h:277-313).
__device__ int cfl_alpha(Smem &sm, const uint8_t *luma, int ls, int startX, int startY, int maxLumaW, int maxLumaH,
                         int log2W, int log2H, int dcv, const uint8_t *sp, int stride, int excludeZero, int *avgOut) {
  int w = 1 << log2W, h = 1 << log2H, n = w * h;
  long long sum = 0;
  for (int k = threadIdx.x; k < n; k += RT) sum += pred::cfl_luma(luma, ls, startX, startY, maxLumaW, maxLumaH, k >> log2W, k & (w - 1));
  int avg = round2((int)cta_sum64(sum, sm), log2W + log2H);
  int sse[33];
  for (int a = 0; a < 33; a++) sse[a] = 0;
  for (int k = threadIdx.x; k < n; k += RT) {
    int i = k >> log2W, j = k & (w - 1);
    int v = pred::cfl_luma(luma, ls, startX, startY, maxLumaW, maxLumaH, i, j) - avg;
    int s0 = sp[i * stride + j];
    for (int a = 0; a < 33; a++) {
      int d = clip3(0, 255, dcv + round2signed((a - 16) * v, 6)) - s0;
      sse[a] += d * d;
    }
  }
  for (int a = threadIdx.x; a < 33; a += RT) sm.sse33[a] = 0;
  __syncthreads();
  for (int a = 0; a < 33; a++) {
    int v = sse[a];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0) atomicAdd(&sm.sse33[a], v);
  }
  __syncthreads();
  long long best = -1;
  int bestA = 0;
  for (int a = -16; a <= 16; a++) {
    if (a == 0 && excludeZero) continue;
    long long s = sm.sse33[a + 16];
    if (best < 0 || s < best) {
      best = s;
      bestA = a;
    }
  }
  __syncthreads();
  *avgOut = avg;
  return bestA;
}

// The clear-flags value of a unit outside the superblock (superblock-relative
// units of the plane, -1..n): clear_block_decoded_flags (k_recon.h:402-414).
__device__ __forceinline__ int decoded_outside(const FrameParams *fp, int r0, int c0, int sub, int y, int x) {
  int n = 16 >> sub;
  if (y == n && x == -1) return 0;
  if (y < 0) return x < ((tile_col_end(fp, c0) - c0) >> sub);
  if (x < 0) return y < ((fp->mi_rows - r0) >> sub);
  return 0;
}

// BlockDecoded of the above-right (k = 0) or below-left (k = 1) corner unit of
// plane p of block b (index me, superblock origin r0, c0) from the frame's
// unit map: the clear-flags value outside the superblock, else whether the
// block covering it precedes this one.
__device__ __forceinline__ int corner_decoded(const FrameParams *fp, const int *blkAt, const BlockInfo &b, int me,
                                              int r0, int c0, int p, int k) {
  int sub = p > 0, n = 16 >> sub;
  int top = (b.mi_row & 15) >> sub, left = (b.mi_col & 15) >> sub;
  int y = k ? top + (block_h(b.bsize) >> (2 + sub)) : top - 1;
  int x = k ? left - 1 : left + (block_w(b.bsize) >> (2 + sub));
  if (y < 0 || x < 0 || y >= n || x >= n) return decoded_outside(fp, r0, c0, sub, y, x);
  int r = r0 + (y << sub), col = c0 + (x << sub);
  if (r >= fp->mi_rows || col >= fp->mi_cols) return 0;
  int blk = blkAt[r * fp->mi_cols + col];
  return blk >= 0 && blk < me;
}

// The edge samples plane p of block b can read : row ay
// from ax0 to ax1 and column x0 - 1 from ly0 to ly1 (empty runs: end <
// start), and the 4x4 luma units under them as two runs (ur, uc, urow, un).
struct EdgeRuns {
  int ay, ax0, ax1, ly0, ly1;
  int ur[2], uc[2], urow[2], un[2];
};
__device__ __forceinline__ EdgeRuns edge_runs(const FrameParams *fp, const BlockInfo &b, int p, int ar, int bl) {
  EdgeRuns e;
  int bs = b.bsize, sub = p > 0, w = block_w(bs) >> sub, h = block_h(bs) >> sub;
  int availU = b.mi_row > 0, availL = b.mi_col > tile_col_start(fp, b.mi_col);
  int x0 = (b.mi_col >> sub) * 4, y0 = (b.mi_row >> sub) * 4;
  int txSz = fp->lossless ? TX_4X4 : sub ? uv_tx_size(bs, 1, 1) : T(Max_Tx_Size_Rect)[bs];
  int ext = imin(T(Tx_Width)[txSz], T(Tx_Height)[txSz]);
  int maxX = ((fp->mi_cols * 4) >> sub) - 1, maxY = ((fp->mi_rows * 4) >> sub) - 1;
  e.ay = y0 - 1;
  e.ax0 = x0 - availL;
  e.ax1 = availU ? imin(maxX, x0 + w - 1 + (ar ? ext : 0)) : e.ax0 - 1;
  e.ly0 = y0 - availU;
  e.ly1 = availL ? imin(maxY, y0 + h - 1 + (bl ? ext : 0)) : e.ly0 - 1;
  e.ur[0] = (e.ay << sub) >> 2;
  e.uc[0] = (e.ax0 << sub) >> 2;
  e.urow[0] = 1;
  e.un[0] = e.ax1 >= e.ax0 ? ((e.ax1 << sub) >> 2) - e.uc[0] + 1 : 0;
  e.ur[1] = (e.ly0 << sub) >> 2;
  e.uc[1] = ((x0 - 1) << sub) >> 2;
  e.urow[1] = 0;
  e.un[1] = e.ly1 >= e.ly0 ? ((e.ly1 << sub) >> 2) - e.ur[1] + 1 : 0;
  return e;
}

// BlockDecoded[plane][y][x] (superblock-relative units of the plane, -1..n)
// as the reference's flags hold it when block sm.blk codes a transform
// block. Outside the superblock: the clear-flags values. Inside, a unit is
// decoded when the block covering it precedes this one in decode order. The
// queries (above-right / below-left of a transform block) land on this
// block itself, directly above it or left of it (blocks there precede it),
// directly right of it or below it (they follow it), or on the block's
// above-right / below-left corner unit, looked up once per block in
// stage_block. `own` answers for a unit of this block: its transform blocks
// run in raster order, so the unit above-right of one is coded (1) and the
// unit below-left is not (0). Units beyond the frame report 0: the edge
// limits clip to maxX / maxY there, so their flag is never used.
__device__ int decoded(const Ctx &c, const Smem &sm, int plane, int y, int x, int own) {
  const FrameParams *fp = c.fp;
  int sub = plane > 0, n = 16 >> sub;
  if (y < 0 || x < 0 || y >= n || x >= n) return decoded_outside(fp, sm.r0, sm.c0, sub, y, x);
  if (sm.r0 + (y << sub) >= fp->mi_rows || sm.c0 + (x << sub) >= fp->mi_cols) return 0;
  const BlockInfo &b = sm.blk;
  int top = (b.mi_row & 15) >> sub, left = (b.mi_col & 15) >> sub;
  int bottom = top + (block_h(b.bsize) >> (2 + sub)), right = left + (block_w(b.bsize) >> (2 + sub));
  if (y >= top && y < bottom && x >= left && x < right) return own;
  if (y == top - 1 && x == right) return sm.cornerAR[plane];
  if (y == bottom && x == left - 1) return sm.cornerBL[plane];
  return y < top || x < left;
}

#define SPIN_LIMIT (1 << 22)  // polls of at least one L2 round trip each: about a second (Ctx::spin_limit)

// A run of 32-bit words to copy from global to shared memory: n words,
// 2^lgw per row, row strides gs (global) / ds (shared) bytes.
struct CopySeg {
  uint8_t *dst;
  const uint8_t *src;
  int ds, gs, n, lgw;
};

// Copies up to NS runs at once through L2 (__ldcg: the frame is being
// written by other SMs): each lane issues the loads of a batch of words
// from any of the runs before its stores, so the whole copy costs about one
// L2 round trip per batch.
#define COPY_BATCH 8
template <int NS>
__device__ void copy_segs(const CopySeg *sg) {
  int total = 0;
#pragma unroll
  for (int k = 0; k < NS; k++) total += sg[k].n;
  for (int base = 0; base < total; base += RT * COPY_BATCH) {
    uint32_t v[COPY_BATCH];
    uint32_t *d[COPY_BATCH];
#pragma unroll
    for (int m = 0; m < COPY_BATCH; m++) {
      int j = base + m * RT + (int)threadIdx.x, k = 0;
      d[m] = nullptr;
      if (j >= total) continue;
#pragma unroll
      for (int q = 0; q < NS - 1; q++)
        if (k == q && j >= sg[q].n) {
          j -= sg[q].n;
          k = q + 1;
        }
      const CopySeg &g = sg[k];
      int r = j >> g.lgw, w = j & ((1 << g.lgw) - 1);
      v[m] = __ldcg((const unsigned *)(g.src + r * g.gs + 4 * w));
      d[m] = (uint32_t *)(g.dst + r * g.ds + 4 * w);
    }
#pragma unroll
    for (int m = 0; m < COPY_BATCH; m++)
      if (d[m]) *d[m] = v[m];
  }
}

// The copies of plane p's edge samples (edge runs e) from frame `from` into
// its tile: the row above from the word holding its first sample, and the
// column left as the word ending at it, one per row. The runs are the union
// of the samples intra_edges reads (above / left limits, spec 7.11.2) over
// every transform block of every candidate size; copies move whole aligned
// words (a word may carry samples no transform block reads).
__device__ __forceinline__ void edge_segs(const Ctx &c, Smem &sm, const uint8_t *from, int p, const EdgeRuns &e, CopySeg *sg) {
  const FrameParams *fp = c.fp;
  const BlockInfo &b = sm.blk;
  int sub = p > 0, S = sub ? TILE_C : TILE_Y;
  uint8_t *t = sub ? sm.tileC[p - 1] : sm.tileY;
  int x0 = (b.mi_col >> sub) * 4, y0 = (b.mi_row >> sub) * 4, fs = fp->stride[p];
  const uint8_t *g = from + fp->offset[p];
  int xs = e.ax0 & ~3;
  sg[0] = CopySeg{t + xs - x0 + TILE_OFF, g + e.ay * fs + xs, 0, 0, e.ax1 >= e.ax0 ? ((e.ax1 - xs) >> 2) + 1 : 0, 20};
  sg[1] = CopySeg{t + (e.ly0 - y0 + 1) * S + TILE_OFF - 4, g + e.ly0 * fs + x0 - 4, S, fs,
                  e.ly1 >= e.ly0 ? e.ly1 - e.ly0 + 1 : 0, 0};
}

// Stages the planes of intra block sm.blk in shared memory, in one
// batch of copies: the block's own samples (the reconstruction so far,
// overwritten as it is coded), its source and its edge samples from frame
// `edges`, complete there. cb: BlockDecoded of its corner units. The views
// then point at the tiles.
__device__ void stage_block(const Ctx &c, Smem &sm, const uint8_t *edges, int cb) {
  const FrameParams *fp = c.fp;
  const BlockInfo &b = sm.blk;
  int bs = b.bsize, tid = threadIdx.x;
  CopySeg sg[4 * 3];
  for (int p = 0; p < 3; p++) {
    int sub = p > 0, S = sub ? TILE_C : TILE_Y, sh = sub ? 2 : 0;
    uint8_t *t = sub ? sm.tileC[p - 1] : sm.tileY, *sb = sub ? sm.srcC[p - 1] : sm.srcY;
    int lw = floor_log2(block_w(bs) >> sub), w = 1 << lw, h = block_h(bs) >> sub;
    int x0 = (b.mi_col >> sub) * 4, y0 = (b.mi_row >> sub) * 4, fs = fp->stride[p];
    sg[4 * p] = CopySeg{t + S + TILE_OFF, c.rec + fp->offset[p] + y0 * fs + x0, S, fs, (w >> 2) * h, lw - 2};
    sg[4 * p + 1] = CopySeg{sb, c.src + fp->offset[p] + y0 * fs + x0, w, fs, (w >> 2) * h, lw - 2};
    edge_segs(c, sm, edges, p, edge_runs(fp, b, p, (cb >> sh) & 1, (cb >> (sh + 1)) & 1), sg + 4 * p + 2);
    if (tid == 0) {
      sm.recp[p] = t + S + TILE_OFF - ((ptrdiff_t)y0 * S + x0);
      sm.rstride[p] = S;
      sm.srcp[p] = sb - ((ptrdiff_t)y0 * w + x0);
      sm.sstride[p] = w;
      sm.cornerAR[p] = (cb >> sh) & 1;
      sm.cornerBL[p] = (cb >> (sh + 1)) & 1;
    }
  }
  copy_segs<4 * 3>(sg);
  __syncthreads();
}

// Writes an intra block's own samples from its tiles
// to the frame (whole words: block positions and widths are multiples of 4
// samples).
__device__ void unstage_intra(const Ctx &c, Smem &sm) {
  const FrameParams *fp = c.fp;
  const BlockInfo &b = sm.blk;
  for (int p = 0; p < 3; p++) {
    int sub = p > 0, S = sub ? TILE_C : TILE_Y;
    const uint8_t *t = sub ? sm.tileC[p - 1] : sm.tileY;
    int lw = floor_log2(block_w(b.bsize) >> sub) - 2, h = block_h(b.bsize) >> sub;
    int x0 = (b.mi_col >> sub) * 4, y0 = (b.mi_row >> sub) * 4, fs = fp->stride[p];
    uint8_t *g = c.rec + fp->offset[p] + y0 * fs + x0;
    for (int k = threadIdx.x; k < (h << lw); k += RT) {
      int i = k >> lw, j = k & ((1 << lw) - 1);
      *(uint32_t *)(g + i * fs + 4 * j) = *(const uint32_t *)(t + (i + 1) * S + TILE_OFF + 4 * j);
    }
  }
}

// Every transform block of one plane of block b (code_plane, k_recon.h:190-291;
// its cost, which no caller here uses, is not summed).
template <bool INTER>
__device__ void code_plane(const Ctx &c, Smem &sm, int plane, int txSz) {
  const FrameParams *fp = c.fp;
  BlockInfo &b = sm.blk;
  int bs = b.bsize, MiRow = b.mi_row, MiCol = b.mi_col;
  int AvailU = MiRow > 0, AvailL = MiCol > tile_col_start(fp, MiCol);
  int sub = plane > 0;
  int planeSz = T(Subsampled_Size)[bs][sub][sub];
  int num4x4W = T(Num_4x4_Blocks_Wide)[planeSz], num4x4H = T(Num_4x4_Blocks_High)[planeSz];
  int baseX = (MiCol >> sub) * 4, baseY = (MiRow >> sub) * 4;
  int stride = sm.sstride[plane];           // source view
  const uint8_t *spx = sm.srcp[plane];
  uint8_t *px = sm.recp[plane];             // reconstruction view
  int rs = sm.rstride[plane];
  int stepX = T(Tx_Width)[txSz] >> 2, stepY = T(Tx_Height)[txSz] >> 2;
  int cands[16], numCands = 0;
  const int isInter = INTER;
  if (plane == 0) {
    int set = get_tx_set(txSz, isInter, fp->reduced_tx_set);
    if (!fp->tx_search || set == TX_SET_DCTONLY || fp->lossless) {
      cands[numCands++] = DCT_DCT;
    } else {
      for (int t = 0; t < 16; t++)
        if (tx_type_in_set(set, t, isInter)) cands[numCands++] = t;
    }
  } else {
    cands[numCands++] = chroma_tx_type(txSz, isInter, b.uv_mode, b.tx_type, fp->reduced_tx_set);
  }
  int txIdx = 0, anyNz = 0;
  int *above = sm.edge[0] + EDGE_OFF, *left = sm.edge[1] + EDGE_OFF, *etmp = sm.edge[2];
  for (int y = 0; y < num4x4H; y += stepY) {
    for (int x = 0; x < num4x4W; x += stepX) {
      int startX = baseX + 4 * x, startY = baseY + 4 * y;
      if (startX >= ((fp->mi_cols * 4) >> sub) || startY >= ((fp->mi_rows * 4) >> sub)) continue;
      int row = (startY << sub) >> 2, col = (startX << sub) >> 2;
      int sbr = row & 15, sbc = col & 15;
      if (!isInter) {
        pred::IntraArgs a;
        a.haveLeft = AvailL || x > 0;
        a.haveAbove = AvailU || y > 0;
        a.haveAboveRight = decoded(c, sm, plane, (sbr >> sub) - 1, (sbc >> sub) + stepX, 1);
        a.haveBelowLeft = decoded(c, sm, plane, (sbr >> sub) + stepY, (sbc >> sub) - 1, 0);
        int isCfl = plane > 0 && b.uv_mode == UV_CFL_PRED;
        a.mode = plane == 0 ? b.y_mode : (isCfl ? DC_PRED : b.uv_mode);
        a.angleDelta = plane == 0 ? b.angle_y : b.angle_uv;
        a.log2W = T(Tx_Width_Log2)[txSz];
        a.log2H = T(Tx_Height_Log2)[txSz];
        a.maxX = ((fp->mi_cols * 4) >> sub) - 1;
        a.maxY = ((fp->mi_rows * 4) >> sub) - 1;
        a.edgeFilter = fp->enable_intra_edge_filter;
        a.filterType = (b.interp_filter >> (plane == 0 ? 4 : 5)) & 1;
        pred::IntraState st;
        pred::intra_state(a, &st);
        pred::intra_edges(px, rs, startX, startY, a, st, above, left, etmp, (int)threadIdx.x, RT, CtaSync());
        int tw = 1 << a.log2W, th = 1 << a.log2H;
        int dcv = a.mode == DC_PRED ? pred::intra_dc(a, above, left) : 0;
        uint8_t *d = px + startY * rs + startX;
        if (threadIdx.x == 0) WORK(W_REC_INTRA_PX, tw * th);
        for (int k = threadIdx.x; k < tw * th; k += RT) {
          int i = k >> a.log2W, j = k & (tw - 1);
          d[i * rs + j] = (uint8_t)(a.mode == DC_PRED ? dcv : pred::intra_pixel(a, st, above, left, i, j));
        }
        __syncthreads();
        if (isCfl) {
          const uint8_t *luma = sm.recp[0];
          int ls = sm.rstride[0];
          int alpha, avg;
          if (txIdx > 0) {
            alpha = plane == 1 ? b.cfl_alpha_u : b.cfl_alpha_v;
            int n = tw * th;
            long long sum = 0;
            for (int k = threadIdx.x; k < n; k += RT)
              sum += pred::cfl_luma(luma, ls, startX, startY, sm.maxLumaW, sm.maxLumaH, k >> a.log2W, k & (tw - 1));
            avg = round2((int)cta_sum64(sum, sm), a.log2W + a.log2H);
          } else {
            alpha = cfl_alpha(sm, luma, ls, startX, startY, sm.maxLumaW, sm.maxLumaH, a.log2W, a.log2H, dcv,
                              spx + startY * stride + startX, stride, plane == 2 && b.cfl_alpha_u == 0, &avg);
            if (threadIdx.x == 0) {
              if (plane == 1) b.cfl_alpha_u = alpha;
              else b.cfl_alpha_v = alpha;
            }
          }
          for (int k = threadIdx.x; k < tw * th; k += RT) {
            int i = k >> a.log2W, j = k & (tw - 1);
            int v = pred::cfl_luma(luma, ls, startX, startY, sm.maxLumaW, sm.maxLumaH, i, j);
            d[i * rs + j] = (uint8_t)pred::cfl_pixel(dcv, alpha, v, avg);
          }
          __syncthreads();
        }
      }
      if (plane == 0 && threadIdx.x == 0) {
        sm.maxLumaW = startX + stepX * 4;
        sm.maxLumaH = startY + stepY * 4;
      }
      int t = DCT_DCT, eob = 0;
      int32_t *coefOut = c.coefs + b.coef_off[plane] + txIdx * T(Tx_Width)[txSz] * T(Tx_Height)[txSz];
      if (fp->lossless) eob = code_wht(c, sm, spx, stride, px, rs, startX, startY, plane, coefOut);
      else if constexpr (INTER)
        eob = code_tx(c, sm, spx, stride, px, rs, startX, startY, txSz, plane, cands, numCands, coefOut, &t);
      if (threadIdx.x == 0 && plane == 0) {
        tx_type_set(b, txIdx, t);
        if (txIdx == 0) b.tx_type = t;
      }
      txIdx++;
      anyNz |= eob > 0;
      __syncthreads();
    }
  }
  if (threadIdx.x == 0) b.eob[plane] = anyNz;
  __syncthreads();
}

// Inter prediction of a w x h block (spec 7.11.3.4) in three steps, staged in
// shared memory: the clamped reference window (h + 7 rows of w + 7 samples),
// the horizontal 8-tap pass of every window row (Round2 by InterRound0 = 3),
// the vertical pass - the values the reference forms sample by sample
// (k_inter.h:451-504). Every tap is even, so half taps (in 8 bits) give the
// same rounded sum: (2 S + 4) >> 3 = (S + 2) >> 2, and a row's 4 sums take 8
// byte dot products on 3 words instead of 32 loads and multiplies; the
// vertical pass slides over 4 rows, 11 loads for 4 samples. Scratch: sm.tmp
// (window), sm.resid (horizontal pass).
constexpr int WIN_P = 80;  // window row pitch: up to 3 samples of alignment, 64 + 7 samples, a word for the last reads
// The window's rows start at win + the returned offset. Inside the picture a
// row is its aligned words; at its borders every sample is clamped.
__device__ __noinline__ int load_window(Smem &sm, const uint8_t *ref, int stride, int lastX, int lastY, int ix0, int iy0, int w, int h) {
  static_assert(sizeof(sm.tmp) >= (64 + 7) * WIN_P, "the window fits its scratch");
  uint8_t *win = (uint8_t *)sm.tmp;
  const int W = w + 7, H = h + 7, lane = threadIdx.x & 31;
  const int off = (int)((uintptr_t)(ref + ix0) & 3);  // rows are multiples of 32 samples apart
  if (ix0 >= 0 && iy0 >= 0 && ix0 + W - 1 <= lastX && iy0 + H - 1 <= lastY) {
    const uint8_t *q = ref + (size_t)iy0 * stride + ix0 - off;
    const int nw = (off + W + 3) >> 2, n = H * nw;
    const unsigned inv = 65535u / nw + 1;  // k / nw for k < 71 * 19
    for (int base = threadIdx.x; base < n; base += 4 * RT) {
      uint32_t v[4];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        int k = base + e * RT, R = (int)(k * inv >> 16);
        if (k < n) v[e] = __ldg((const uint32_t *)(q + (size_t)R * stride) + (k - R * nw));
      }
#pragma unroll
      for (int e = 0; e < 4; e++) {
        int k = base + e * RT, R = (int)(k * inv >> 16);
        if (k < n) *(uint32_t *)(win + R * WIN_P + 4 * (k - R * nw)) = v[e];
      }
    }
  } else {
    for (int R = threadIdx.x >> 5; R < H; R += RT / 32) {
      const uint8_t *row = ref + (size_t)clip3(0, lastY, iy0 + R) * stride;
      for (int C = lane; C < W; C += 32) win[R * WIN_P + off + C] = __ldg(row + clip3(0, lastX, ix0 + C));
    }
  }
  __syncthreads();
  return off;
}
__device__ __forceinline__ int dp4(uint32_t px, int taps, int acc) {
  int r;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(px), "r"(taps), "r"(acc));
  return r;
}
__device__ __noinline__ void horizontal_pass(Smem &sm, int off, const int16_t *fh, int lw, int h) {
  const uint8_t *win = (const uint8_t *)sm.tmp;
  int16_t *hs = (int16_t *)sm.resid;
  int t0 = 0, t1 = 0;
  for (int t = 0; t < 4; t++) {
    t0 |= ((fh[t] >> 1) & 255) << (8 * t);
    t1 |= ((fh[t + 4] >> 1) & 255) << (8 * t);
  }
  const int lq = lw - 2, n = (h + 7) << lq;
  for (int k = threadIdx.x; k < n; k += RT) {
    int R = k >> lq, c = (k & ((1 << lq) - 1)) * 4;
    const uint32_t *q = (const uint32_t *)(win + R * WIN_P + c);
    // samples c .. c + 11 of the row, aligned
    uint32_t a = __funnelshift_r(q[0], q[1], 8 * off), b = __funnelshift_r(q[1], q[2], 8 * off), d = __funnelshift_r(q[2], q[3], 8 * off);
    int s0 = (dp4(b, t1, dp4(a, t0, 2))) >> 2;
    int s1 = (dp4(__funnelshift_r(b, d, 8), t1, dp4(__funnelshift_r(a, b, 8), t0, 2))) >> 2;
    int s2 = (dp4(__funnelshift_r(b, d, 16), t1, dp4(__funnelshift_r(a, b, 16), t0, 2))) >> 2;
    int s3 = (dp4(__funnelshift_r(b, d, 24), t1, dp4(__funnelshift_r(a, b, 24), t0, 2))) >> 2;
    *(uint2 *)(hs + (R << lw) + c) = make_uint2((s0 & 0xffff) | (uint32_t)s1 << 16, (s2 & 0xffff) | (uint32_t)s3 << 16);
  }
  __syncthreads();
}
// The vertical pass; out(row, column, sum before its rounding).
template <class Out>
__device__ __forceinline__ void vertical_pass(Smem &sm, const int16_t *fv, int lw, int h, Out out) {
  const int16_t *hs = (const int16_t *)sm.resid;
  const int w = 1 << lw, n = (h >> 2) << lw;
  int f[8];
  for (int t = 0; t < 8; t++) f[t] = fv[t];
  for (int k = threadIdx.x; k < n; k += RT) {
    int r = (k >> lw) * 4, c = k & (w - 1);
    int v[11];
#pragma unroll
    for (int t = 0; t < 11; t++) v[t] = hs[((r + t) << lw) + c];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      int acc = 0;
#pragma unroll
      for (int t = 0; t < 8; t++) acc += f[t] * v[q + t];
      out(r + q, c, acc);
    }
  }
}
// mode 0: final samples (Round2 by 11, clipped) into d (stride ds); 1:
// compound intermediates (Round2 by 7) into sm.pred0; 2: Round2(pred0 + this
// block's intermediates, 5), clipped, into d.
__device__ __noinline__ void predict_block(Smem &sm, const pred::Inter &ip, int lw, int h, int mode, uint8_t *d, int ds) {
  if (threadIdx.x == 0) WORK(W_REC_INTER_PX, h << lw);
  const int off = load_window(sm, ip.ref, ip.stride, ip.lastX, ip.lastY, ip.ix0, ip.iy0, 1 << lw, h);
  horizontal_pass(sm, off, ip.fh, lw, h);
  if (mode == 0)
    vertical_pass(sm, ip.fv, lw, h, [&](int r, int c, int acc) { d[r * ds + c] = (uint8_t)clip1(round2(acc, 11)); });
  else if (mode == 1)
    vertical_pass(sm, ip.fv, lw, h, [&](int r, int c, int acc) { sm.pred0[(r << lw) + c] = (int16_t)round2(acc, 7); });
  else
    vertical_pass(sm, ip.fv, lw, h, [&](int r, int c, int acc) {
      d[r * ds + c] = (uint8_t)clip1(round2((int)sm.pred0[(r << lw) + c] + round2(acc, 7), 5));
    });
  __syncthreads();
}


// ---- bulk copies (the TMA engine's cp.async.bulk) into shared memory ------------------
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

// One row copy global -> shared, completing on the mbarrier: both addresses
// 16-byte aligned, bytes a multiple of 16 (checked by the caller's layout).
__device__ __forceinline__ void bulk_row(void *dst, const void *src, unsigned bytes, unsigned long long *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// Waits (bounded) for phase `parity` of the mbarrier to complete; false if
// it did not within `limit` polls.
__device__ __forceinline__ bool bar_wait(unsigned long long *bar, unsigned parity, int limit) {
  for (int i = 0; i < limit; i++) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// The superblock's source (luma 64 rows of 64 bytes, two chroma planes of
// 32 rows of 32 bytes) into sm.srcSB: one bulk copy per row, a thread each,
// all completing on sm.bar's phase. Rows are 16-byte aligned in the padded frame
// layout (luma stride sb_cols * 64, chroma sb_cols * 32, superblock columns
// at multiples of 64 / 32 bytes, plane offsets multiples of 64). On a wait
// past the limit the error and abort words are set (status 4) and the copies
// are waited for again before the CTA goes on, so none lands after it.
__device__ void stage_sb_source(const Ctx &c, Smem &sm, int sb, unsigned phase) {
  static_assert(INTER_THREADS == 128, "one thread per source row");
  const FrameParams *fp = c.fp;
  int sbr = sb / fp->sb_cols, sbc = sb % fp->sb_cols, t = threadIdx.x;
  if (t == 0) {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    // the previous block's reads of the tile come before the copies into it
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&sm.bar)),
                 "r"(64 * 64 + 2 * 32 * 32)
                 : "memory");
  }
  __syncthreads();
  if (t < 64) {
    bulk_row(sm.srcSB + t * 64, c.src + fp->offset[0] + (size_t)(sbr * 64 + t) * fp->stride[0] + sbc * 64, 64, &sm.bar);
  } else {
    int p = 1 + ((t - 64) >> 5), r = (t - 64) & 31;
    bulk_row(sm.srcSB + 64 * 64 + (p - 1) * 32 * 32 + r * 32,
             c.src + fp->offset[p] + (size_t)(sbr * 32 + r) * fp->stride[p] + sbc * 32, 32, &sm.bar);
  }
  if (!bar_wait(&sm.bar, phase, c.spin_limit)) {
    if (t == 0) {
      atomicExch(c.status, 4);
      atomicExch(c.status + 1, 1);
    }
    bar_wait(&sm.bar, phase, c.spin_limit);
  }
}

// The inter block's plane p: views of the staged source (absolute plane
// coordinates into sm.srcSB) and of sm.recT (the block's own w x h samples).
__device__ __forceinline__ void inter_views(const Ctx &c, Smem &sm, int p) {
  const BlockInfo &b = sm.blk;
  int sub = p > 0, S = sub ? 32 : 64;
  int sbx = (sm.c0 * 4) >> sub, sby = (sm.r0 * 4) >> sub;
  const uint8_t *tile = sm.srcSB + (sub ? 64 * 64 + (p - 1) * 32 * 32 : 0);
  int w = block_w(b.bsize) >> sub, x0 = (b.mi_col >> sub) * 4, y0 = (b.mi_row >> sub) * 4;
  sm.srcp[p] = tile - ((ptrdiff_t)sby * S + sbx);
  sm.sstride[p] = S;
  sm.recp[p] = sm.recT - ((ptrdiff_t)y0 * w + x0);
  sm.rstride[p] = w;
}

// Writes plane p of the inter block back from sm.recT to the frame (whole
// words: block positions and widths are multiples of 4 samples).
__device__ void unstage_inter(const Ctx &c, Smem &sm, int p) {
  const FrameParams *fp = c.fp;
  const BlockInfo &b = sm.blk;
  int sub = p > 0, lw = floor_log2(block_w(b.bsize) >> sub) - 2, h = block_h(b.bsize) >> sub;
  int x0 = (b.mi_col >> sub) * 4, y0 = (b.mi_row >> sub) * 4, fs = fp->stride[p];
  uint8_t *g = c.rec + fp->offset[p] + y0 * fs + x0;
  for (int k = threadIdx.x; k < (h << lw); k += RT) {
    int i = k >> lw, j = k & ((1 << lw) - 1);
    *(uint32_t *)(g + i * fs + 4 * j) = *(const uint32_t *)(sm.recT + (i << (lw + 2)) + 4 * j);
  }
  __syncthreads();
}

// The dual interpolation filter search of a single-reference block
// (k_recon.h:304-328): sm.blk's interp_filter.
__device__ __noinline__ void filter_search(const Ctx &c, Smem &sm, const uint8_t *ref) {
  const FrameParams *fp = c.fp;
  BlockInfo &b = sm.blk;
  const int bs = b.bsize, MiRow = b.mi_row, MiCol = b.mi_col, tid = threadIdx.x;
  int w = block_w(bs), h = block_h(bs);
  int x0 = MiCol * 4, y0 = MiRow * 4, stride = fp->stride[0], ss = sm.sstride[0];
  const uint8_t *sp = sm.srcp[0] + y0 * ss + x0;
  int vw = imin(w, fp->frame_w - x0), vh = imin(h, fp->frame_h - y0);
  long long best = -1;
  int bestPacked = 0, off = 0;
  // the window once, a horizontal pass per horizontal filter, a vertical
  // pass with its SSE per pair
  for (int fh = 0; fh < 3; fh++)
    for (int fv = 0; fv < 3; fv++) {
      int packed = fv | (fh << 2);
      pred::Inter ip;
      pred::inter_setup(&ip, ref + fp->offset[0], stride, fp->frame_w, fp->frame_h, x0, y0, w, h, b.mv_row, b.mv_col,
                        0, 0, packed);
      if (fh == 0 && fv == 0) off = load_window(sm, ip.ref, ip.stride, ip.lastX, ip.lastY, ip.ix0, ip.iy0, w, h);
      if (fv == 0) horizontal_pass(sm, off, ip.fh, floor_log2(w), h);
      if (tid == 0) WORK(W_REC_INTER_PX, w * h);
      int sse = 0;  // at most 32 samples of 255^2 a thread
      vertical_pass(sm, ip.fv, floor_log2(w), h, [&](int r, int c, int acc) {
        if (r < vh && c < vw) {
          int d = clip1(round2(acc, 11)) - (int)sp[r * ss + c];
          sse += d * d;
        }
      });
      long long cst = cta_sum64(sse, sm) * 16 + (long long)fp->lambda * ((fv != 0) + (fh != 0));
      if (best < 0 || cst < best) {
        best = cst;
        bestPacked = packed;
      }
    }
  if (tid == 0) b.interp_filter = bestPacked;
  __syncthreads();
}

// One inter block (recon_block, k_recon.h:293-394); sm.blk holds it. Its
// planes are coded in sm.recT one after another, each written back after it.
__device__ void recon_inter_block(const Ctx &c, Smem &sm, BlockInfo *gb) {
  const FrameParams *fp = c.fp;
  BlockInfo &b = sm.blk;
  int bs = b.bsize;
  int comp = b.ref_frame1 > INTRA_FRAME;
  const uint8_t *ref = b.ref_frame != LAST_FRAME ? c.gold : c.ref;
  const uint8_t *ref1 = c.gold;
  const int MiRow = b.mi_row, MiCol = b.mi_col;
  if (threadIdx.x == 0) {
    sm.maxLumaW = sm.maxLumaH = 0;
    b.tx_depth = 0;
    b.interp_filter &= 0x30;
  }
  if (threadIdx.x < 3) inter_views(c, sm, threadIdx.x);
  __syncthreads();
  int tid = threadIdx.x;
  if (fp->switchable_interp && !comp) filter_search(c, sm, ref);
  for (int plane = 0; plane < 3; plane++) {
    int sub = plane > 0, stride = fp->stride[plane];
    int baseX = (MiCol >> sub) * 4, baseY = (MiRow >> sub) * 4;
    int w = block_w(bs) >> sub, h = block_h(bs) >> sub;
    int rs = sm.rstride[plane];
    uint8_t *d = sm.recp[plane] + baseY * rs + baseX;
    pred::Inter p0, p1;
    pred::inter_setup(&p0, ref + fp->offset[plane], stride, fp->frame_w, fp->frame_h, baseX, baseY, w, h, b.mv_row,
                      b.mv_col, sub, sub, b.interp_filter);
    if (comp)
      pred::inter_setup(&p1, ref1 + fp->offset[plane], stride, fp->frame_w, fp->frame_h, baseX, baseY, w, h,
                        b.mv1_row, b.mv1_col, sub, sub, b.interp_filter);
    if (comp) {
      predict_block(sm, p0, floor_log2(w), h, 1, d, rs);
      predict_block(sm, p1, floor_log2(w), h, 2, d, rs);
    } else {
      predict_block(sm, p0, floor_log2(w), h, 0, d, rs);
    }
    code_plane<true>(c, sm, plane,
                     fp->lossless ? TX_4X4 : plane > 0 ? uv_tx_size(bs, 1, 1) : T(Max_Tx_Size_Rect)[bs]);
    unstage_inter(c, sm, plane);
  }
  if (tid == 0) *gb = b;
}

// The CTA's shared copies of the frame parameters and the quantiser's
// reciprocals; returns the context reading them.
__device__ Ctx load_shared(const Ctx &c, Smem &sm) {
  const int *src = (const int *)c.fp;
  int *dst = (int *)&sm.fpc;
  for (int k = threadIdx.x; k < (int)(sizeof(FrameParams) / 4); k += RT) dst[k] = src[k];
  Ctx cs = c;
  cs.fp = &sm.fpc;
  // the reciprocals are 64-bit divisions: once per CTA, not per transform block
  if (threadIdx.x < 6) {
    int p = threadIdx.x >> 1, q = (threadIdx.x & 1) ? c.fp->ac_q[p] : c.fp->dc_q[p];
    sm.qinv[p][threadIdx.x & 1] = q > 0 ? tx::quant_inv(q) : 0;
  }
  __syncthreads();
  return cs;
}

// The inter blocks of the frame (they read reference pictures only, so none
// waits): persistent CTAs take them from the list, large ones first. With one
// CTA per superblock the frame took as long as its most divided superblock
// (2.4 ms for a 640x360 full-tool frame's 60, half of it now); CTAs assigned
// by slot cost a 3840x2160 leaf frame 80 us in CTAs without a block.
__global__ void __launch_bounds__(INTER_THREADS, 512 / INTER_THREADS) k_recon_inter(Ctx cg) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem &sm = *(Smem *)smem_raw;
  const int big = cg.counters[CNT_BIG], total = big + cg.counters[CNT_SMALL], tid = threadIdx.x;
  if ((int)blockIdx.x >= total) return;
  const Ctx c = load_shared(cg, sm);
  if (tid == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sm.bar)) : "memory");
  for (unsigned phase = 0;; phase ^= 1) {
    if (tid == 0) sm.flag = atomicAdd(c.counters + CNT_TAKEN, 1);
    __syncthreads();
    const int k = sm.flag;
    if (k >= total) return;
    const int me = c.inter[k < big ? k : c.nblk - 1 - (k - big)], sb = me / MAX_BLOCKS_PER_SB;
    if (tid == 32) {
      sm.r0 = (sb / c.fp->sb_cols) * 16;
      sm.c0 = (sb % c.fp->sb_cols) * 16;
    }
    if (tid < (int)(sizeof(BlockInfo) / 4)) ((int *)&sm.blk)[tid] = ((const int *)(c.blocks + me))[tid];
    stage_sb_source(c, sm, sb, phase);
    __syncthreads();
    recon_inter_block(c, sm, c.blocks + me);
    __syncthreads();
  }
}

// ---- the intra blocks --------------------------------------------------------------------
//
// Luma and chroma of a block are separate tasks of one dataflow. A block's
// luma may run once the luma of every intra block under its edges is written;
// its chroma once its own luma and those blocks' chroma are (both planes' edge
// samples lie over the same neighbours, so one successor list serves both
// chains). Each kind has its own workers, ready queue and counters, so neither
// chain waits in the other's code, and a worker whose block was some
// successor's last dependency goes on with that successor itself: the chain's
// step has no queue in it. A step used to take about 24,500 cycles for an 8x8
// block's luma (descriptor 2,100, staging 4,500, edges and prediction 6,000,
// transforms 6,100, publishing 3,700), chroma as much behind it; the chain is
// some 650 blocks deep on a 1080p key frame, so the step is the frame's time.
//
// What depends only on the block is worked out for all blocks at once by the
// prepass (k_block_deps): place, transform, edge limits, filter and upsampling
// decisions, in one 128-byte record.
struct PlaneTask {
  int x, y;      // first sample, plane coordinates
  unsigned geo;  // log2 w | log2 h << 3 | mode << 6 | haveLeft << 10 | haveAbove << 11 | upAbove << 12 | upLeft << 13
                 // | strengthAbove << 14 | strengthLeft << 16 | corner filter << 18 | cfl << 19 | tx type << 20 | tx size << 24
  unsigned lim;  // samples available above | left << 16 (at least 1 each)
  unsigned flt;  // samples the edge filter covers, above | left << 16 (the corner included)
  unsigned ang;  // pAngle | dx << 9 | dy << 20
};
struct IntraTask {
  int me, nsucc;
  int coef[3];
  int interp;                // interp_filter & 0x30
  int bits;                  // BlockDecoded of the corner units: bit 0 / 1 luma above-right / below-left, bit 2 / 3 chroma
  int maxLumaW, maxLumaH;    // CfL's luma limits
  PlaneTask p[2];            // luma, chroma
  int angle_y, bsize;
  int pad[9];
};
static_assert(sizeof(IntraTask) == 128, "one coalesced load of a warp");

// Everything about plane `sub` of block b coded as one transform block (an
// intra block of at most 64x64 without a transform split).
__device__ PlaneTask plane_task(const FrameParams *fp, const BlockInfo &b, int sub, int ar, int bl) {
  PlaneTask t;
  int bs = b.bsize, lw = floor_log2(block_w(bs) >> sub), lh = floor_log2(block_h(bs) >> sub), w = 1 << lw, h = 1 << lh;
  int haveLeft = b.mi_col > tile_col_start(fp, b.mi_col), haveAbove = b.mi_row > 0;
  t.x = (b.mi_col >> sub) * 4;
  t.y = (b.mi_row >> sub) * 4;
  int maxX = ((fp->mi_cols * 4) >> sub) - 1, maxY = ((fp->mi_rows * 4) >> sub) - 1;
  int isCfl = sub && b.uv_mode == UV_CFL_PRED;
  pred::IntraArgs a;
  a.mode = !sub ? b.y_mode : isCfl ? DC_PRED : b.uv_mode;
  a.angleDelta = sub ? b.angle_uv : b.angle_y;
  a.log2W = lw;
  a.log2H = lh;
  a.edgeFilter = fp->enable_intra_edge_filter;
  a.filterType = (b.interp_filter >> (4 + sub)) & 1;
  pred::IntraState st;
  pred::intra_state(a, &st);
  int sa = 0, sl = 0, corner = 0, za = 0, zl = 0;
  if (intra_is_directional(a.mode) && a.edgeFilter && st.pAngle != 90 && st.pAngle != 180) {
    corner = st.pAngle > 90 && st.pAngle < 180 && w + h >= 24;
    if (haveAbove) sa = pred::edge_strength(w, h, a.filterType, st.pAngle - 90);
    if (haveLeft) sl = pred::edge_strength(w, h, a.filterType, st.pAngle - 180);
    za = imin(w, maxX - t.x + 1) + (st.pAngle < 90 ? h : 0) + 1;
    zl = imin(h, maxY - t.y + 1) + (st.pAngle > 180 ? w : 0) + 1;
  }
  int txSz = sub ? uv_tx_size(bs, 1, 1) : T(Max_Tx_Size_Rect)[bs];
  int type = sub ? chroma_tx_type(txSz, 0, b.uv_mode, 0, fp->reduced_tx_set) : DCT_DCT;
  t.geo = (unsigned)(lw | lh << 3 | a.mode << 6 | haveLeft << 10 | haveAbove << 11 | st.upAbove << 12 | st.upLeft << 13 |
                     sa << 14 | sl << 16 | corner << 18 | isCfl << 19 | type << 20 | txSz << 24);
  t.lim = (unsigned)(imin(maxX, t.x + (ar ? 2 * w : w) - 1) - t.x + 1) |
          (unsigned)(imin(maxY, t.y + (bl ? 2 * h : h) - 1) - t.y + 1) << 16;
  t.flt = (unsigned)(za | zl << 16);
  t.ang = (unsigned)(st.pAngle | st.dx << 9) | (unsigned)st.dy << 20;
  return t;
}

// Per frame, before the recon launches: the block index of every 4x4 luma
// unit of the frame, the list of inter blocks and the number of intra blocks
// (a CTA per superblock, a warp per block, its lanes over the block's units).
constexpr int MAP_THREADS = 256;
__global__ void __launch_bounds__(MAP_THREADS) k_block_map(const FrameParams *fp, const BlockInfo *blocks, const SbInfo *sbs, int *blkAt,
                                                  int *counters, int *inter, int nblk) {
  int sb = blockIdx.x, lane = threadIdx.x & 31, intra = 0;
  int cols = fp->mi_cols, rows = fp->mi_rows, n = imin(sbs[sb].num_blocks, MAX_BLOCKS_PER_SB);
  for (int k = threadIdx.x >> 5; k < n; k += MAP_THREADS / 32) {
    int idx = sb * MAX_BLOCKS_PER_SB + k;
    const BlockInfo &b = blocks[idx];
    if (!b.is_inter) {
      intra++;
    } else if (lane == 0) {
      if (block_w(b.bsize) * block_h(b.bsize) >= 32 * 32) inter[atomicAdd(counters + CNT_BIG, 1)] = idx;
      else inter[nblk - 1 - atomicAdd(counters + CNT_SMALL, 1)] = idx;
    }
    if (b.mi_row < 0 || b.mi_col < 0) continue;
    int h = imax(0, imin(T(Num_4x4_Blocks_High)[b.bsize], rows - b.mi_row));
    int lw = floor_log2(T(Num_4x4_Blocks_Wide)[b.bsize]), w = imax(0, imin(1 << lw, cols - b.mi_col));
    for (int i = lane; i < h << lw; i += 32) {
      int r = i >> lw, c = i & ((1 << lw) - 1);
      if (c < w) blkAt[(b.mi_row + r) * cols + b.mi_col + c] = idx;
    }
  }
  if (lane == 0 && intra) atomicAdd(counters + CNT_TOTAL, intra);
}

// Orders this thread's (and, after a barrier, its CTA's) accesses before it
// with those after it, at device scope.
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Appends a block to a ready queue (kind 0: luma, 1: chroma). What the caller
// knows complete, it has ordered before by a fence (or an earlier launch).
__device__ __forceinline__ void push_ready(const Ctx &c, int kind, int blk) {
  int t = atomicAdd(c.counters + CNT_TAIL + kind, 1);
  atomicExch(c.queue + kind * c.nblk + t, blk + 1);
}

// Per frame, after the unit map, one warp per block slot: each intra block's
// record and its dependencies. The blocks under its luma and chroma edge
// samples (edge_runs with its corner units' BlockDecoded) that are intra and
// not itself, without repeats: their number is its luma dependency count (and
// with its own luma its chroma count), and it joins each one's successor
// list. Blocks with none start in the luma queue.
__global__ void __launch_bounds__(128) k_block_deps(Ctx c) {
  __shared__ int cand[4][160];
  const FrameParams *fp = c.fp;
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, me = blockIdx.x * 4 + warp;
  if (me >= c.nblk) return;
  int sb = me / MAX_BLOCKS_PER_SB;
  if (me % MAX_BLOCKS_PER_SB >= c.sbs[sb].num_blocks) return;
  BlockInfo b = c.blocks[me];
  if (b.is_inter) return;
  int r0 = (sb / fp->sb_cols) * 16, c0 = (sb % fp->sb_cols) * 16;
  EdgeRuns e[2];  // luma; chroma (both chroma planes share their geometry)
  int cb = 0;
  for (int p = 0; p < 2; p++) {
    int ar = corner_decoded(fp, c.blk_at, b, me, r0, c0, p, 0), bl = corner_decoded(fp, c.blk_at, b, me, r0, c0, p, 1);
    e[p] = edge_runs(fp, b, p, ar, bl);
    cb |= (ar | bl << 1) << (2 * p);
  }
  IntraTask *task = c.tasks + me;
  if (lane < 2) task->p[lane] = plane_task(fp, b, lane, (cb >> (2 * lane)) & 1, (cb >> (2 * lane + 1)) & 1);
  if (lane == 2) {
    task->me = me;
    for (int p = 0; p < 3; p++) task->coef[p] = b.coef_off[p];
    task->interp = b.interp_filter & 0x30;
    task->bits = cb;
    task->angle_y = b.angle_y;
    task->bsize = b.bsize;
    task->maxLumaW = b.mi_col * 4 + block_w(b.bsize);
    task->maxLumaH = b.mi_row * 4 + block_h(b.bsize);
  }
  int run[4] = {e[0].un[0], e[0].un[1], e[1].un[0], e[1].un[1]};
  int n = imin(160, run[0] + run[1] + run[2] + run[3]);
  for (int i = lane; i < n; i += 32) {
    int k = 0, j = i;
    while (j >= run[k]) j -= run[k++];
    const EdgeRuns &er = e[k >> 1];
    int kk = k & 1;
    int r = er.ur[kk] + (er.urow[kk] ? 0 : j), col = er.uc[kk] + (er.urow[kk] ? j : 0);
    int d = c.blk_at[r * fp->mi_cols + col];
    if (d == me || (unsigned)d >= (unsigned)c.nblk || c.blocks[d].is_inter) d = -1;
    cand[warp][i] = d;
  }
  __syncwarp();
  int cnt = 0;
  for (int i = lane; i < n; i += 32) {
    int d = cand[warp][i];
    if (d < 0) continue;
    bool dup = false;
    for (int j = 0; j < i && !dup; j++) dup = cand[warp][j] == d;
    if (dup) continue;
    cnt++;
    int slot = atomicAdd(c.succ_count + d, 1);
    if (slot < MAX_SUCC) {
      c.succ[(size_t)d * MAX_SUCC + slot] = me;
    } else {
      atomicExch(c.status, 2);
      atomicExch(c.status + 1, 1);
    }
  }
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  if (lane == 0) {
    c.dep_count[c.nblk + me] = cnt + 1;
    cnt += me == c.hold;
    if (cnt == 0) push_ready(c, 0, me);
    else c.dep_count[me] = cnt;
  }
}

// Threads of one plane: NT of them, ranks 0 .. NT - 1, with a named barrier.
template <int NT>
struct Group {
  int tid, bar;
  __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(NT) : "memory"); }
  __device__ __forceinline__ int any(int p) const {
    int r;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.s32 p, %1, 0;\n bar.red.or.pred q, %2, %3, p;\n selp.s32 %0, 1, 0, q;\n}\n"
        : "=r"(r)
        : "r"(p), "r"(bar), "n"(NT)
        : "memory");
    return r;
  }
};

// Working memory of a plane of at most MAXD x MAXD samples.
template <int MAXD>
struct PlaneMem {
  // residual, then the inverse transform's rows: 16-byte aligned and 4 banks apart (8 rows a lane each meet no bank twice)
  __align__(16) int32_t resid[MAXD * (MAXD + 4)];
  int32_t tmp[MAXD * 32];            // forward row pass; before it CfL's luma values
  int32_t q[32 * 32];
  int32_t lv[MAXD == 64 ? 32 * 32 : 1];  // levels, where they are read again (code_large)
  int edge[4][EDGE_LEN];             // AboveRow, LeftCol, filter copies of both
  __align__(4) uint8_t px[MAXD * MAXD];  // prediction, then reconstruction (stride w)
  int sse[8][33];
  int red[8], alpha;
};
struct IntraShared {
  FrameParams fpc;
  uint64_t qinv[3][2];
  int32_t fmat[3][FMAT_SMALL], fmatT[3][FMAT_SMALL];
  int smw[124];      // smooth weights of lengths 4, 8, 16, 32, 64 from (1 << log2) - 4
  IntraTask task;
  int coded;         // the coders are past the block's last stores (feed)
  int alphaU;        // U's CfL alpha
  union {
    PlaneMem<64> y;
    PlaneMem<32> uv[2];
  };
};

// What a prediction does to its edges, and a directional mode's slopes.
struct EdgePrep {
  int pAngle, dx, dy, upA, upL;  // pred::IntraState
  int sa, sl, corner, za, zl;    // filter strengths (0: none), the corner filter, samples covered (the corner included)
};

// Edge filter (7.11.2.12) and upsampling (7.11.2.11) of a block's edges, both
// sides at once.
template <int NT>
__device__ __forceinline__ void prepare_edges(const Group<NT> &g, const EdgePrep &e, int *above, int *left, int *ta, int *tl, int w,
                                              int h) {
  const int tid = g.tid;
  if (e.corner | e.sa | e.sl) {
    const int za = e.sa ? e.za : 0, zl = e.sl ? e.zl : 0;
    if (e.corner) {
      if (tid == 0) left[-1] = above[-1] = round2(left[0] * 5 + above[-1] * 6 + above[0] * 5, 4);
      g.sync();
    }
    if (za | zl) {
      for (int i = tid; i < za + zl; i += NT) {
        if (i < za) ta[i] = above[i - 1];
        else tl[i - za] = left[i - za - 1];
      }
      g.sync();
      for (int i = tid; i < za + zl; i += NT) {
        int a = i < za, k = a ? i : i - za, z = a ? za : zl, s = a ? e.sa : e.sl;
        const int *src = a ? ta : tl;
        if (k == 0) continue;
        int acc = 0;
        for (int j = 0; j < 5; j++) acc += T(Intra_Edge_Kernel)[s - 1][j] * src[clip3(0, z - 1, k - 2 + j)];
        (a ? above : left)[k - 1] = (acc + 8) >> 4;
      }
      g.sync();
    }
  }
  if (e.upA | e.upL) {
    const int nA = e.upA ? w + (e.pAngle < 90 ? h : 0) : 0, nL = e.upL ? h + (e.pAngle > 180 ? w : 0) : 0;
    const int cA = e.upA ? nA + 3 : 0, cL = e.upL ? nL + 3 : 0;
    for (int i = tid; i < cA + cL; i += NT) {
      int a = i < cA, k = a ? i : i - cA, n = a ? nA : nL;
      (a ? ta : tl)[k] = (a ? above : left)[k == 0 ? -1 : imin(k - 2, n - 1)];
    }
    g.sync();
    for (int i = tid; i < nA + nL; i += NT) {
      int a = i < nA, k = a ? i : i - nA;
      const int *d = (a ? ta : tl) + k;
      int *buf = a ? above : left;
      buf[2 * k - 1] = clip1(round2(-d[0] + 9 * d[1] + 9 * d[2] - d[3], 4));
      buf[2 * k] = d[2];
      if (k == 0) buf[-2] = d[0];
    }
    g.sync();
  }
}

// DC_PRED's value (pred::intra_dc), by every warp for itself.
__device__ __forceinline__ int dc_value(const int *above, const int *left, int lw, int lh, int haveAbove, int haveLeft) {
  const int w = 1 << lw, h = 1 << lh, lane = threadIdx.x & 31;
  int sA = 0, sL = 0;
  for (int i = lane; i < w; i += 32) sA += above[i];
  for (int i = lane; i < h; i += 32) sL += left[i];
  sA = __reduce_add_sync(0xffffffffu, sA);
  sL = __reduce_add_sync(0xffffffffu, sL);
  if (haveLeft && haveAbove) return (sA + sL + ((w + h) >> 1)) / (w + h);
  if (haveLeft) return (sL + (h >> 1)) >> lh;
  if (haveAbove) return (sA + (w >> 1)) >> lw;
  return 128;
}

// Samples (i, j0 .. j0 + 3) of a w x h prediction from prepared edges
// (pred::intra_pixel; wX, wY: smooth weights of w and h).
__device__ __forceinline__ void predict4(int mode, const EdgePrep &e, const int *above, const int *left, const int *wX, const int *wY,
                                         int w, int h, int i, int j0, int dcv, int (&p)[4]) {
  const int upA = e.upA, upL = e.upL, dx = e.dx, dy = e.dy;
  if (mode == DC_PRED) {
    for (int k = 0; k < 4; k++) p[k] = dcv;
  } else if (intra_is_directional(mode)) {
    if (e.pAngle < 90) {
      int idx = (i + 1) * dx, shift = ((idx << upA) >> 1) & 0x1F, b0 = (idx >> (6 - upA)) + (j0 << upA), mx = (w + h - 1) << upA;
      for (int k = 0; k < 4; k++) {
        int b = b0 + (k << upA);
        p[k] = b < mx ? round2(above[b] * (32 - shift) + above[b + 1] * shift, 5) : above[mx];
      }
    } else if (e.pAngle > 90 && e.pAngle < 180) {
      for (int k = 0; k < 4; k++) {
        int j = j0 + k, idx = (j << 6) - (i + 1) * dx, b = idx >> (6 - upA), up = upA;
        const int *ed = above;
        if (b < -(1 << upA)) {
          idx = (i << 6) - (j + 1) * dy;
          b = idx >> (6 - upL);
          ed = left;
          up = upL;
        }
        int shift = ((idx * (1 << up)) >> 1) & 0x1F;
        p[k] = round2(ed[b] * (32 - shift) + ed[b + 1] * shift, 5);
      }
    } else if (e.pAngle > 180) {
      for (int k = 0; k < 4; k++) {
        int idx = (j0 + k + 1) * dy, b = (idx >> (6 - upL)) + (i << upL), shift = ((idx << upL) >> 1) & 0x1F;
        p[k] = round2(left[b] * (32 - shift) + left[b + 1] * shift, 5);
      }
    } else if (e.pAngle == 90) {
      for (int k = 0; k < 4; k++) p[k] = above[j0 + k];
    } else {
      for (int k = 0; k < 4; k++) p[k] = left[i];
    }
  } else if (mode == PAETH_PRED) {
    int L = left[i], C = above[-1];
    for (int k = 0; k < 4; k++) {
      int A = above[j0 + k], base = A + L - C, pl = iabs(base - L), pt = iabs(base - A), pc = iabs(base - C);
      p[k] = pl <= pt && pl <= pc ? L : pt <= pc ? A : C;
    }
  } else {  // SMOOTH, SMOOTH_V, SMOOTH_H
    int L = left[i], LB = left[h - 1], AR = above[w - 1], wy = wY[i];
    for (int k = 0; k < 4; k++) {
      int A = above[j0 + k], wx = wX[j0 + k];
      int v = wy * A + (256 - wy) * LB, hh = wx * L + (256 - wx) * AR;
      p[k] = mode == SMOOTH_PRED ? round2(v + hh, 9) : mode == SMOOTH_V_PRED ? round2(v, 8) : round2(hh, 8);
    }
  }
}

// Inverse transform of the dequantised levels in m.q, added into m.px.
template <int MAXD, int NT, int HIGH>
__device__ __forceinline__ void inverse_g(PlaneMem<MAXD> &m, const Group<NT> &g, int lw, int lh, int type, int txSz, int dcQ, int acQ) {
  constexpr int RS = MAXD + 4;
  const int w = 1 << lw, h = 1 << lh, th = imin(32, h), rowShift = T(Transform_Row_Shift)[txSz], denom = tx::dq_denom(txSz);
  const int rect = iabs(lw - lh) == 1, rk = tx::row_kind(type), ck = tx::col_kind(type);
  if (HIGH >= 5 && lw >= 5) {
    for (int p = g.tid; p < 2 * h; p += NT) {
      if (lw == 5) inv_row_split<5, RS, false>(m.resid, m.q, p >> 1, p & 1, th, dcQ, acQ, denom, rect, rowShift);
      else if (HIGH >= 6) inv_row_split<6, RS, false>(m.resid, m.q, p >> 1, p & 1, th, dcQ, acQ, denom, rect, rowShift);
    }
  } else {
    for (int i = g.tid; i < h; i += NT) {
      if (lw == 2) inv_row<2, RS, false>(m.resid, m.q, i, th, dcQ, acQ, denom, rect, rk, rowShift);
      else if (lw == 3) inv_row<3, RS, false>(m.resid, m.q, i, th, dcQ, acQ, denom, rect, rk, rowShift);
      else if (lw == 4) inv_row<4, RS, false>(m.resid, m.q, i, th, dcQ, acQ, denom, rect, rk, rowShift);
    }
  }
  g.sync();
  if (HIGH >= 5 && lh >= 5) {
    for (int p = g.tid; p < 2 * w; p += NT) {
      if (lh == 5) inv_col_split<5, RS>(m.resid, p >> 1, p & 1, w, 0, 0, m.px, w, 0, 0);
      else if (HIGH >= 6) inv_col_split<6, RS>(m.resid, p >> 1, p & 1, w, 0, 0, m.px, w, 0, 0);
    }
  } else {
    for (int j = g.tid; j < w; j += NT) {
      if (lh == 2) inv_col<2, RS>(m.resid, j, w, ck, 0, 0, m.px, w, 0, 0);
      else if (lh == 3) inv_col<3, RS>(m.resid, j, w, ck, 0, 0, m.px, w, 0, 0);
      else if (lh == 4) inv_col<4, RS>(m.resid, j, w, ck, 0, 0, m.px, w, 0, 0);
    }
  }
  g.sync();
}
// Lengths above 16 are DCT in an intra block (TX_SET_DCTONLY). Out of line:
// the common sizes' registers do not carry the 32- and 64-point kernels.
template <int MAXD, int NT>
__device__ __noinline__ void inverse_large(PlaneMem<MAXD> &m, const Group<NT> g, int lw, int lh, int type, int txSz, int dcQ, int acQ) {
  inverse_g<MAXD, NT, MAXD == 64 ? 6 : 5>(m, g, lw, lh, type, txSz, dcQ, acQ);
}

// CfL prediction of a chroma plane (spec 7.11.5; cfl_best_alpha,
// k_intra.h:277-313): the luma average, the first least SSE over alpha in
// [-16, 16] against the source (`sv`, this thread's source words), the
// prediction into m.px. V waits for U's alpha: 0 is excluded when U's is 0.
// Up to 32 samples a lane takes an alpha and runs over the samples; above,
// a thread takes samples, 33 sums each.
template <int MAXD, int NT, int MAXW>
__device__ __forceinline__ void cfl_g(const Ctx &c, IntraShared &sh, PlaneMem<MAXD> &m, const Group<NT> &g, const PlaneTask &t,
                                      int plane, int dcv, const uint32_t (&sv)[MAXW]) {
  const int lw = t.geo & 7, lh = (t.geo >> 3) & 7, w = 1 << lw, n = 1 << (lw + lh), lane = g.tid & 31, warp = g.tid >> 5;
  const FrameParams *fp = &sh.fpc;
  const uint8_t *luma = c.rec + fp->offset[0];
  const int ls = fp->stride[0], mw = sh.task.maxLumaW, mh = sh.task.maxLumaH;
  int *lv = m.tmp;  // luma value per sample | source sample << 16
  int sum = 0;
#pragma unroll
  for (int q = 0; q < MAXW; q++) {
    int k = (g.tid + q * NT) * 4;
    if (k >= n) break;
    int i = k >> lw, j = k & (w - 1);
    int ly = imin((t.y + i) << 1, mh - 2);
    const uint8_t *l0 = luma + (size_t)ly * ls;
    unsigned short a[4], b[4];
    for (int e = 0; e < 4; e++) {
      int lx = imin((t.x + j + e) << 1, mw - 2);  // even: the pair is one 16-bit word
      a[e] = __ldcg((const unsigned short *)(l0 + lx));
      b[e] = __ldcg((const unsigned short *)(l0 + ls + lx));
    }
    for (int e = 0; e < 4; e++) {
      int v = ((a[e] & 255) + (a[e] >> 8) + (b[e] & 255) + (b[e] >> 8)) << 1;
      lv[k + e] = v | (int)((sv[q] >> (8 * e)) & 255) << 16;
      sum += v;
    }
  }
  sum = __reduce_add_sync(0xffffffffu, sum);
  if (lane == 0) m.red[warp] = sum;
  g.sync();
  sum = 0;
  for (int k = 0; k < NT / 32; k++) sum += m.red[k];
  const int avg = round2(sum, lw + lh);
  if (n <= 32) {
    if (warp == 0) {
      int s = 0;
      for (int k = 0; k < n; k++) {
        int x = lv[k], d = clip3(0, 255, dcv + round2signed((lane - 16) * ((x & 0xffff) - avg), 6)) - (x >> 16);
        s += d * d;
      }
      m.sse[0][lane] = s;
    } else if (warp == 1) {
      int s = 0;
      if (lane < n) {
        int x = lv[lane], d = clip3(0, 255, dcv + round2signed(16 * ((x & 0xffff) - avg), 6)) - (x >> 16);
        s = d * d;
      }
      s = __reduce_add_sync(0xffffffffu, s);
      if (lane == 0) m.sse[0][32] = s;
    }
  } else {
    int s[33];
#pragma unroll
    for (int a = 0; a < 33; a++) s[a] = 0;
    for (int k = g.tid; k < n; k += NT) {
      int x = lv[k], v = (x & 0xffff) - avg, s0 = x >> 16;
#pragma unroll
      for (int a = 0; a < 33; a++) {
        int d = clip3(0, 255, dcv + round2signed((a - 16) * v, 6)) - s0;
        s[a] += d * d;
      }
    }
    int mine = 0, last = 0;
#pragma unroll
    for (int a = 0; a < 33; a++) {
      int r = __reduce_add_sync(0xffffffffu, s[a]);
      if (a == lane) mine = r;
      if (a == 32) last = r;
    }
    m.sse[warp][lane] = mine;
    if (lane == 0) m.sse[warp][32] = last;
  }
  g.sync();
  if (plane == 2) asm volatile("bar.sync 3, %0;" ::"n"(2 * NT) : "memory");  // U's alpha
  if (warp == 0) {
    int s = 0, s32 = 0;
    const int parts = n <= 32 ? 1 : NT / 32;
    for (int k = 0; k < parts; k++) {
      s += m.sse[k][lane];
      s32 += m.sse[k][32];
    }
    if (plane == 2 && sh.alphaU == 0 && lane == 16) s = 0x7fffffff;
    int best = __reduce_min_sync(0xffffffffu, s);
    int at = __ffs(__ballot_sync(0xffffffffu, s == best)) - 1;
    if (s32 < best) at = 32;
    if (lane == 0) {
      m.alpha = at - 16;
      if (plane == 1) sh.alphaU = at - 16;
    }
  }
  if (plane == 1) asm volatile("bar.sync 3, %0;" ::"n"(2 * NT) : "memory");
  g.sync();
  const int alpha = m.alpha;
  for (int k = g.tid; k < n; k += NT) m.px[k] = (uint8_t)pred::cfl_pixel(dcv, alpha, lv[k] & 0xffff, avg);
}

// One plane of an intra block as one transform block with one type: edges
// from the frame (through L2: other SMs write it during the launch),
// prediction, forward transform, quantiser, inverse, reconstruction written to
// the frame (code_plane / code_tx_block, k_recon.h:60-291). The whole group
// calls it; the frame's words are written when it returns, without a barrier.
// Returns whether the block has levels.
template <int MAXD, int NT>
__device__ __forceinline__ int code_single(const Ctx &c, IntraShared &sh, PlaneMem<MAXD> &m, const Group<NT> g, const PlaneTask &t,
                                           int plane) {
  constexpr int RS = MAXD + 4, MAXW = MAXD * MAXD / 4 / NT;
  const FrameParams *fp = &sh.fpc;
  const int tid = g.tid;
  const unsigned geo = t.geo;
  const int lw = geo & 7, lh = (geo >> 3) & 7, w = 1 << lw, h = 1 << lh, wl = lw - 2, nw = 1 << (lw + lh - 2);
  const int mode = (geo >> 6) & 15, haveLeft = (geo >> 10) & 1, haveAbove = (geo >> 11) & 1;
  const int stride = fp->stride[plane];
  const size_t o = fp->offset[plane] + (size_t)t.y * stride + t.x;
  const uint8_t *sp = c.src + o;
  uint8_t *rp = c.rec + o;
  uint32_t sv[MAXW];
#pragma unroll
  for (int q = 0; q < MAXW; q++) {
    int k = tid + q * NT;
    if (k < nw) sv[q] = __ldg((const uint32_t *)(sp + (k >> wl) * stride) + (k & ((1 << wl) - 1)));
  }
  int *above = m.edge[0] + EDGE_OFF, *left = m.edge[1] + EDGE_OFF, *ta = m.edge[2], *tl = m.edge[3];
  {  // AboveRow, LeftCol and the corner (spec 7.11.2)
    const int n = w + h, nA = t.lim & 0xffff, nL = t.lim >> 16;
    for (int i = tid; i < 2 * n + 1; i += NT) {
      int v, *to;
      if (i < n) {
        to = above + i;
        v = haveAbove ? ldpx(rp - stride + imin(i, nA - 1)) : haveLeft ? ldpx(rp - 1) : 127;
      } else if (i < 2 * n) {
        to = left + i - n;
        v = haveLeft ? ldpx(rp + imin(i - n, nL - 1) * stride - 1) : haveAbove ? ldpx(rp - stride) : 129;
      } else {
        to = above - 1;
        v = haveAbove && haveLeft ? ldpx(rp - stride - 1) : haveAbove ? ldpx(rp - stride) : haveLeft ? ldpx(rp - 1) : 128;
        left[-1] = v;
      }
      *to = v;
    }
  }
  g.sync();
  const EdgePrep e = {(int)(t.ang & 511), (int)((t.ang >> 9) & 2047), (int)(t.ang >> 20), (int)((geo >> 12) & 1), (int)((geo >> 13) & 1),
                      (int)((geo >> 14) & 3), (int)((geo >> 16) & 3), (int)((geo >> 18) & 1), (int)(t.flt & 0xffff), (int)(t.flt >> 16)};
  prepare_edges(g, e, above, left, ta, tl, w, h);
  const int dcv = mode == DC_PRED ? dc_value(above, left, lw, lh, haveAbove, haveLeft) : 0;
  const int cfl = plane && ((geo >> 19) & 1);
  if (cfl) {
    if constexpr (MAXD == 32) cfl_g(c, sh, m, g, t, plane, dcv, sv);
    g.sync();
  }
  if (tid == 0) WORK(W_REC_INTRA_PX, w * h);
  // prediction and residual, a word of 4 samples at a time
  const int *wX = sh.smw + w - 4, *wY = sh.smw + h - 4;
#pragma unroll
  for (int q = 0; q < MAXW; q++) {
    int k = tid + q * NT;
    if (k >= nw) break;
    int i = k >> wl, j0 = (k & ((1 << wl) - 1)) * 4;
    int p[4];
    if (cfl) {
      uint32_t v = *(const uint32_t *)(m.px + 4 * k);
      for (int k4 = 0; k4 < 4; k4++) p[k4] = (v >> (8 * k4)) & 255;
    } else {
      predict4(mode, e, above, left, wX, wY, w, h, i, j0, dcv, p);
    }
    uint32_t pk = 0;
    int32_t *rr = m.resid + i * RS + j0;
#pragma unroll
    for (int k4 = 0; k4 < 4; k4++) {
      pk |= (uint32_t)(p[k4] & 255) << (8 * k4);
      rr[k4] = (int)((sv[q] >> (8 * k4)) & 255) - p[k4];
    }
    *(uint32_t *)(m.px + 4 * k) = pk;
  }
  g.sync();
  // forward transform and quantiser
  const int type = (geo >> 20) & 15, txSz = (geo >> 24) & 31;
  const int tw = imin(32, w), th = imin(32, h), ltw = imin(5, lw), dcQ = fp->dc_q[plane], acQ = fp->ac_q[plane];
  const int rk = tx::row_kind(type), ck = tx::col_kind(type);
  const int32_t *Mh = lw <= 4 ? sh.fmatT[rk] + (lw == 2 ? 0 : lw == 3 ? 16 : 80) : c.mats_t + fwd_slot(rk, lw);
  const int32_t *Mv = lh <= 4 ? sh.fmat[ck] + (lh == 2 ? 0 : lh == 3 ? 16 : 80) : c.mats + fwd_slot(ck, lh);
  if (tid == 0) {
    WORK(W_REC_FWD_MAC, h * tw * w + th * tw * h);
    WORK(W_REC_QUANT, th * tw);
  }
  fwd_rows_any<RS>(lw, m.resid, m.tmp, Mh, h, tid, NT);
  g.sync();
  const int shifts = T(Transform_Row_Shift)[txSz] + 4, rect = iabs(lw - lh) == 1, denom = tx::dq_denom(txSz);
  const uint64_t invDc = sh.qinv[plane][0], invAc = sh.qinv[plane][1];
  int32_t *coefOut = c.coefs + sh.task.coef[plane];
  int nz = 0;
  fwd_cols_any(lh, m.tmp, Mv, ltw, tid, NT, [&](int k, int64_t s) {
    int first = k == 0;
    int lv = tx::quant_level(fwd_scale(s, shifts, rect), first ? dcQ : acQ, first ? 26 : 22, denom, first ? invDc : invAc);
    m.q[k] = tx::dequant_level(lv, first ? dcQ : acQ, denom);
    coefOut[k] = lv;
    nz |= lv;
  });
  nz = g.any(nz);
  if (nz) {
    if (tid == 0) WORK(W_REC_INV_OPS, 3 * (1 << (lw + lh)) * (lw + lh));
    if (lw <= 4 && lh <= 4) inverse_g<MAXD, NT, 4>(m, g, lw, lh, type, txSz, dcQ, acQ);
    else inverse_large<MAXD, NT>(m, g, lw, lh, type, txSz, dcQ, acQ);
  }
#pragma unroll
  for (int q = 0; q < MAXW; q++) {
    int k = tid + q * NT;
    if (k < nw) *((uint32_t *)(rp + (k >> wl) * stride) + (k & ((1 << wl) - 1))) = *(const uint32_t *)(m.px + 4 * k);
  }
  return nz;
}

// The workers' shared constants.
template <class Shared>
__device__ void load_intra_shared(const Ctx &c, Shared &sh) {
  const int nt = blockDim.x;
  for (int k = threadIdx.x; k < (int)(sizeof(FrameParams) / 4); k += nt) ((int *)&sh.fpc)[k] = ((const int *)c.fp)[k];
  if (threadIdx.x < 6) {
    int p = threadIdx.x >> 1, q = (threadIdx.x & 1) ? c.fp->ac_q[p] : c.fp->dc_q[p];
    sh.qinv[p][threadIdx.x & 1] = q > 0 ? tx::quant_inv(q) : 0;
  }
  for (int kind = 0; kind < 3; kind++)
    for (int lg = 2; lg <= 4; lg++) {
      int n = 1 << (2 * lg), off = lg == 2 ? 0 : lg == 3 ? 16 : 80;
      for (int k = threadIdx.x; k < n; k += nt) {
        sh.fmat[kind][off + k] = c.mats[fwd_slot(kind, lg) + k];
        sh.fmatT[kind][off + k] = c.mats_t[fwd_slot(kind, lg) + k];
      }
    }
  for (int k = threadIdx.x; k < 124; k += nt)
    sh.smw[k] = k < 4 ? T(Sm_Weights_Tx_4x4)[k] : k < 12 ? T(Sm_Weights_Tx_8x8)[k - 4] : k < 28 ? T(Sm_Weights_Tx_16x16)[k - 12]
                : k < 60 ? T(Sm_Weights_Tx_32x32)[k - 28] : T(Sm_Weights_Tx_64x64)[k - 60];
  __syncthreads();
}

// The next block of a ready queue (one thread): its slot is claimed, then
// waited for (bounded) until a released block fills it; -1 once every block
// of the kind is done, or after a wait somewhere gave up.
__device__ int pop_ready(const Ctx &c, int kind, int total) {
  volatile int *abort = c.status + 1, *done = c.counters + CNT_DONE + kind;
  if (*abort) return -1;
  int slot = atomicAdd(c.counters + CNT_HEAD + kind, 1);
  if (slot >= total) return -1;
  volatile int *vslot = c.queue + kind * c.nblk + slot;
  for (int spins = 0;; spins++) {
    int v = *vslot, d = *done;
    if (v) {
      fence_gpu();
      return v - 1;
    }
    if (d >= total || *abort) return -1;
    if (spins > c.spin_limit) {
      atomicExch(c.status, 1);
      atomicExch(c.status + 1, 1);
      return -1;
    }
    __nanosleep(32);
  }
}

// A worker CTA's last warp: it takes blocks, loads their records for the
// coding warps and releases successors, so that queue traffic runs beside the
// coding. Barrier 4: the record is in place (me -1: no more); barrier 5: the
// block is coded and written.
//
// While a block is coded the warp watches its successors' dependency counts: a
// successor with one dependency left waits for this block alone, so it is the
// next block whatever else happens, and its record is fetched at once. When
// the block is coded the coding warps go on with it after two barriers, and
// only then are the other successors released, with the fence and the atomics
// that takes (about 3,000 cycles that used to lie between two blocks of a
// chain, of 10,000). Otherwise the first successor that this block's release
// makes ready follows.
constexpr int CODERS = 128, WORKER_THREADS = CODERS + 32;
template <int N>
__device__ __forceinline__ void record_bar() { asm volatile("bar.sync 4, %0;" ::"n"(N) : "memory"); }
template <int N>
__device__ __forceinline__ void coded_bar() { asm volatile("bar.sync 5, %0;" ::"n"(N) : "memory"); }

template <int N, class Shared>
__device__ void feed(const Ctx &c, Shared &sh, int kind, int total) {
  const int lane = threadIdx.x & 31;
  volatile int *coded = &sh.coded;
  int *dep = c.dep_count + kind * c.nblk;
  auto record_word = [&](int b) {
    return __ldcg(lane == 1 ? c.succ_count + b : (const int *)(c.tasks + b) + lane);
  };
  int s[3] = {-1, -1, -1};  // this lane's successors of the block being coded, or of `prev`
  int push[3] = {-1, -1, -1}, own = -1;  // ready blocks still to be queued: successors, the block's own chroma (lane 0)
  int prev = -1;                         // a block coded but not yet released, all but its successor `me`
  for (int me = -1, word = 0;;) {
    if (me < 0) {
      if (lane == 0) me = pop_ready(c, kind, total);
      me = __shfl_sync(0xffffffffu, me, 0);
      if (me >= 0) word = record_word(me);
    }
    ((int *)&sh.task)[lane] = me < 0 ? -1 : word;
    if (lane == 0) *coded = 0;
    __syncwarp();
    record_bar<N>();
    if (me < 0) return;
    const int n = imin(__shfl_sync(0xffffffffu, word, 1), MAX_SUCC);
    if (prev >= 0) {
      fence_gpu();
      int left[3], mine = 0;
#pragma unroll
      for (int q = 0; q < 3; q++) left[q] = s[q] >= 0 && s[q] != me ? atomicSub(dep + s[q], 1) : 0;
      if (kind == 0 && lane == 0) mine = atomicSub(c.dep_count + c.nblk + prev, 1);
#pragma unroll
      for (int q = 0; q < 3; q++) push[q] = left[q] == 1 ? s[q] : -1;
      own = mine == 1 ? prev : -1;
      fence_gpu();
      if (lane == 0) atomicAdd(c.counters + CNT_DONE + kind, 1);
      prev = -1;
    }
    // the successors and the pending queue entries, in flight together
#pragma unroll
    for (int q = 0; q < 3; q++) s[q] = lane + 32 * q < n ? __ldcg(c.succ + (size_t)me * MAX_SUCC + lane + 32 * q) : -1;
    {
      int t[3] = {0, 0, 0}, town = 0;
      if (own >= 0) town = atomicAdd(c.counters + CNT_TAIL + 1, 1);
#pragma unroll
      for (int q = 0; q < 3; q++)
        if (push[q] >= 0) t[q] = atomicAdd(c.counters + CNT_TAIL + kind, 1);
      if (own >= 0) atomicExch(c.queue + c.nblk + town, own + 1);
#pragma unroll
      for (int q = 0; q < 3; q++)
        if (push[q] >= 0) atomicExch(c.queue + kind * c.nblk + t[q], push[q] + 1);
    }
    // (what the watch misses, the release below finds: its limit only ends the look-ahead)
    int next = -1;
    const unsigned r = watch_ready(FullWarp(), c.spin_limit, [&] { return *coded != 0; },
                                   [&] { return s[0] >= 0 && *(volatile int *)(dep + imax(s[0], 0)) == 1; });
    if (r) {
      fence_gpu();  // what its other dependencies wrote is visible, its record among it
      next = __shfl_sync(0xffffffffu, s[0], __ffs(r) - 1);
      word = record_word(next);
    }
    __syncwarp();
    coded_bar<N>();
    if (next >= 0) {
      prev = me;
      me = next;
      push[0] = push[1] = push[2] = own = -1;
      continue;
    }
    fence_gpu();
    int left[3], mine = 0;
#pragma unroll
    for (int q = 0; q < 3; q++) left[q] = s[q] >= 0 ? atomicSub(dep + s[q], 1) : 0;
    if (kind == 0 && lane == 0) mine = atomicSub(c.dep_count + c.nblk + me, 1);
    own = mine == 1 ? me : -1;
#pragma unroll
    for (int q = 0; q < 3; q++) {
      int ready = left[q] == 1;
      unsigned r = __ballot_sync(0xffffffffu, ready);
      if (next < 0 && r) {
        int f = __ffs(r) - 1;
        next = __shfl_sync(0xffffffffu, s[q], f);
        if (lane == f) ready = 0;
      }
      push[q] = ready ? s[q] : -1;
    }
    // what the other dependencies wrote is visible to the coders (and to whoever takes a queued block)
    fence_gpu();
    if (lane == 0) atomicAdd(c.counters + CNT_DONE + kind, 1);
    me = next;
    if (me >= 0) {
      word = record_word(me);
    } else {  // nothing to go on with: queue the chroma before waiting
      if (own >= 0) push_ready(c, 1, own);
      own = -1;
    }
  }
}

// Workers per kind: as many as the frame's blocks can use, so that on frames
// of few intra blocks the other SMs stay free for the other engine's kernels.
#ifndef MAV1CU_BLOCKS_PER_WORKER
#define MAV1CU_BLOCKS_PER_WORKER 16
#endif
#ifndef MAV1CU_MIN_WORKERS
#define MAV1CU_MIN_WORKERS 8
#endif
constexpr int BLOCKS_PER_WORKER = MAV1CU_BLOCKS_PER_WORKER, MIN_WORKERS = MAV1CU_MIN_WORKERS;

// ---- workers of frames whose luma blocks are one transform block of one type (no
// transform type or depth search, not lossless)
__device__ void luma_worker(const Ctx &c, IntraShared &sh) {
  const Group<CODERS> g{(int)threadIdx.x, 1};
  for (;;) {
    record_bar<WORKER_THREADS>();
    const int me = sh.task.me;
    if (me < 0) return;
    const int nz = code_single<64, CODERS>(c, sh, sh.y, g, sh.task.p[0], 0);
    if (g.tid == CODERS - 1) {
      BlockInfo *gb = c.blocks + me;
      gb->tx_depth = 0;
      gb->interp_filter = sh.task.interp;
      gb->tx_type = DCT_DCT;
      gb->tx_types_lo &= ~15;
      gb->eob[0] = nz;
    }
    if (g.tid == 0) *(volatile int *)&sh.coded = 1;
    coded_bar<WORKER_THREADS>();
  }
}

// Chroma: U and V at once, half of the coding warps each.
__device__ void chroma_worker(const Ctx &c, IntraShared &sh) {
  constexpr int NT = CODERS / 2;
  const int plane = 1 + (int)threadIdx.x / NT;
  const Group<NT> g{(int)threadIdx.x % NT, plane};
  PlaneMem<32> &m = sh.uv[plane - 1];
  for (;;) {
    record_bar<WORKER_THREADS>();
    const int me = sh.task.me;
    if (me < 0) return;
    const int nz = code_single<32, NT>(c, sh, m, g, sh.task.p[1], plane);
    if (g.tid == NT - 1) {
      BlockInfo *gb = c.blocks + me;
      gb->eob[plane] = nz;
      if ((sh.task.p[1].geo >> 19) & 1) (plane == 1 ? gb->cfl_alpha_u : gb->cfl_alpha_v) = m.alpha;
    }
    if (threadIdx.x == 0) *(volatile int *)&sh.coded = 1;
    coded_bar<WORKER_THREADS>();
  }
}

// ---- luma with the transform type and depth searches ---------------------------------------
//
// The candidates of a transform block do not depend on one another: a warp
// takes each (at most 7 types up to 16 x 16, DCT alone above), with its own
// scratch, and the least cost is chosen after one barrier. The depths follow
// one another, every one from the same pixels; the best one's pixels, types
// and levels are kept when a later depth overwrites them, instead of coding it
// again. A transform block's candidates used to run one after another on the
// whole CTA, 11,000 cycles each with ten barriers, for every depth and once
// more for the winner.
constexpr int SEARCH_CODERS = 256, SEARCH_WORKERS = SEARCH_CODERS + 32;
struct SearchShared {
  FrameParams fpc;
  uint64_t qinv[3][2];
  int32_t fmat[3][FMAT_SMALL], fmatT[3][FMAT_SMALL];
  int smw[124];
  IntraTask task;
  int coded;
  long long cost[8];
  int eob[8];
  long long red[8];
  int lo, hi, type0, anyNz, maxW, maxH;  // the block's tx_types, tx_type, eob[0], CfL limits as coded so far
  int bestTypes[16], types[16], bestN, bestNz, bestW, bestH;
  int above[132], left[132];             // the block's edges from the corner at [0]
  __align__(4) uint8_t px[64 * 64], best[64 * 64], src[64 * 64];  // stride 64
  int32_t bestCoef[64 * 64];
  union {
    PlaneMem<64> m;
    Cand cand[SEARCH_CODERS / 32];
  };
};

// One candidate type in a warp: eval's result for candidate ci.
__device__ __forceinline__ void eval_candidate(SearchShared &sh, Cand &cd, int ci, int type, int txSz, int x, int y, int lane) {
  const FrameParams *fp = &sh.fpc;
  const int lw = T(Tx_Width_Log2)[txSz], lh = T(Tx_Height_Log2)[txSz], rk = tx::row_kind(type), ck = tx::col_kind(type);
  const CandIn in = {sh.src + y * 64 + x, sh.px + y * 64 + x, 64, 64,
                     sh.fmatT[rk] + (lw == 2 ? 0 : lw == 3 ? 16 : 80), sh.fmat[ck] + (lh == 2 ? 0 : lh == 3 ? 16 : 80),
                     fp->dc_q[0], fp->ac_q[0], sh.qinv[0][0], sh.qinv[0][1], fp->lambda};
  int eob;
  long long cost = cand_cost(in, cd, type, txSz, lane, &eob);
  if (lane == 0) {
    sh.cost[ci] = cost;
    sh.eob[ci] = eob;
  }
}

__device__ __forceinline__ long long group_sum(SearchShared &sh, const Group<SEARCH_CODERS> &g, long long v) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  g.sync();
  if ((g.tid & 31) == 0) sh.red[g.tid >> 5] = v;
  g.sync();
  v = 0;
  for (int k = 0; k < SEARCH_CODERS / 32; k++) v += sh.red[k];
  return v;
}

// A transform block with a length above 16 (DCT alone): the group's threads
// together; its reconstruction goes to sh.px, its levels to coefOut. Returns
// the cost; *eobOut the eob.
__device__ __noinline__ long long code_large(const Ctx &c, SearchShared &sh, const Group<SEARCH_CODERS> g, int txSz, int x, int y,
                                             int32_t *coefOut, int *eobOut) {
  const FrameParams *fp = &sh.fpc;
  PlaneMem<64> &m = sh.m;
  constexpr int NT = SEARCH_CODERS, RS = 68;
  const int tid = g.tid, lw = T(Tx_Width_Log2)[txSz], lh = T(Tx_Height_Log2)[txSz], w = 1 << lw, h = 1 << lh;
  const int tw = imin(32, w), th = imin(32, h), ltw = imin(5, lw);
  for (int k = tid; k < w * h; k += NT) {
    int i = k >> lw, j = k & (w - 1), p = sh.px[(y + i) * 64 + x + j];
    m.px[k] = (uint8_t)p;
    m.resid[i * RS + j] = (int)sh.src[(y + i) * 64 + x + j] - p;
  }
  g.sync();
  const int32_t *Mh = lw <= 4 ? sh.fmatT[0] + (lw == 2 ? 0 : lw == 3 ? 16 : 80) : c.mats_t + fwd_slot(0, lw);
  const int32_t *Mv = lh <= 4 ? sh.fmat[0] + (lh == 2 ? 0 : lh == 3 ? 16 : 80) : c.mats + fwd_slot(0, lh);
  if (tid == 0) {
    WORK(W_REC_FWD_MAC, h * tw * w + th * tw * h);
    WORK(W_REC_QUANT, th * tw);
  }
  fwd_rows_any<RS>(lw, m.resid, m.tmp, Mh, h, tid, NT);
  g.sync();
  const int dcQ = fp->dc_q[0], acQ = fp->ac_q[0], shifts = T(Transform_Row_Shift)[txSz] + 4, rect = iabs(lw - lh) == 1;
  const int denom = tx::dq_denom(txSz);
  const uint64_t invDc = sh.qinv[0][0], invAc = sh.qinv[0][1];
  const int16_t *inv = d_inv_scan + d_inv_scan_off[0][txSz];
  int eob = 0;
  fwd_cols_any(lh, m.tmp, Mv, ltw, tid, NT, [&](int k, int64_t s) {
    int first = k == 0;
    int lv = tx::quant_level(fwd_scale(s, shifts, rect), first ? dcQ : acQ, first ? 26 : 22, denom, first ? invDc : invAc);
    m.q[k] = tx::dequant_level(lv, first ? dcQ : acQ, denom);
    m.lv[k] = lv;
    coefOut[k] = lv;
    if (lv) eob = imax(eob, inv[k] + 1);
  });
  eob = __reduce_max_sync(0xffffffffu, eob);
  if ((tid & 31) == 0) sh.eob[tid >> 5] = eob;
  g.sync();
  for (int k = 0; k < NT / 32; k++) eob = imax(eob, sh.eob[k]);
  long long bits = 0, sse = 0;
  if (eob == 0) {
    bits = tid == 0 ? 8 : 0;
  } else {
    for (int k = tid; k < th * tw; k += NT)
      if (inv[k] < eob) bits += level_bits(m.lv[k]);
    if (tid == 0) bits += 8 * 6 + 8 * 2 * (31 - __clz(eob + 1));
    if (tid == 0) WORK(W_REC_INV_OPS, 3 * (1 << (lw + lh)) * (lw + lh));
    inverse_large<64, NT>(m, g, lw, lh, DCT_DCT, txSz, dcQ, acQ);
  }
  for (int k = tid; k < w * h; k += NT) {
    int i = k >> lw, j = k & (w - 1), v = m.px[k];
    int d = (int)sh.src[(y + i) * 64 + x + j] - v;
    sse += d * d;
    sh.px[(y + i) * 64 + x + j] = (uint8_t)v;
  }
  sse = group_sum(sh, g, sse);
  bits = group_sum(sh, g, bits);
  *eobOut = eob;
  return sse * 16 + (long long)fp->lambda * bits / 8;
}

// The block's luma at one transform size (code_plane, k_recon.h:190-291):
// returns the cost. sh.types lists the transform blocks' types, *nTx their number.
__device__ long long code_depth(const Ctx &c, SearchShared &sh, const Group<SEARCH_CODERS> &g, int txSz, int *nTx) {
  const FrameParams *fp = &sh.fpc;
  const PlaneTask &t = sh.task.p[0];
  const int tid = g.tid, lane = tid & 31, warp = tid >> 5;
  const unsigned geo = t.geo;
  const int bw = 1 << (geo & 7), bh = 1 << ((geo >> 3) & 7), mode = (geo >> 6) & 15;
  const int lw = T(Tx_Width_Log2)[txSz], lh = T(Tx_Height_Log2)[txSz], w = 1 << lw, h = 1 << lh;
  const int maxX = fp->mi_cols * 4 - 1, maxY = fp->mi_rows * 4 - 1;
  const int set = get_tx_set(txSz, 0, fp->reduced_tx_set);
  unsigned cands = 0;  // types, a nibble each, in the set's order
  int numCands = 0;
  if (!fp->tx_search || set == TX_SET_DCTONLY) {
    numCands = 1;
  } else {
    for (int k = 0; k < 16; k++)
      if (tx_type_in_set(set, k, 0)) cands |= (unsigned)k << (4 * numCands++);
  }
  pred::IntraArgs ia;
  ia.mode = mode;
  ia.angleDelta = sh.task.angle_y;
  ia.log2W = lw;
  ia.log2H = lh;
  ia.edgeFilter = fp->enable_intra_edge_filter;
  ia.filterType = (sh.task.interp >> 4) & 1;
  pred::IntraState st;
  pred::intra_state(ia, &st);
  EdgePrep e = {st.pAngle, st.dx, st.dy, st.upAbove, st.upLeft, 0, 0, 0, 0, 0};
  const bool filtered = intra_is_directional(mode) && ia.edgeFilter && st.pAngle != 90 && st.pAngle != 180;
  PlaneMem<64> &m = sh.m;
  // the edge arrays lie behind the candidates' scratch
  static_assert(offsetof(PlaneMem<64>, edge) >= sizeof(Cand) * (SEARCH_CODERS / 32), "edges and candidates overlap");
  int *above = m.edge[0] + EDGE_OFF, *left = m.edge[1] + EDGE_OFF;
  long long total = 0;
  int idx = 0;
  for (int y = 0; y < bh; y += h)
    for (int x = 0; x < bw; x += w) {
      const int X = t.x + x, Y = t.y + y;
      if (X > maxX || Y > maxY) continue;
      const int haveLeft = ((geo >> 10) & 1) || x > 0, haveAbove = ((geo >> 11) & 1) || y > 0;
      const int ar = y == 0 ? (x + w == bw ? sh.task.bits & 1 : 1) : x + w < bw;
      const int bl = x == 0 ? (y + h == bh ? (sh.task.bits >> 1) & 1 : 1) : 0;
      {
        const int n = w + h, nA = imin(maxX, X + (ar ? 2 * w : w) - 1) - X + 1, nL = imin(maxY, Y + (bl ? 2 * h : h) - 1) - Y + 1;
        // sample (x + dx, y - 1) / (x - 1, y + dy) of the block: its own pixels or its edges
        auto up = [&](int d) { return y > 0 && (x > 0 || d >= 0) ? (int)sh.px[(y - 1) * 64 + x + d] : y > 0 ? sh.left[y] : sh.above[x + d + 1]; };
        auto lf = [&](int d) { return x > 0 ? (int)sh.px[(y + d) * 64 + x - 1] : sh.left[y + d + 1]; };
        for (int i = tid; i < 2 * n + 1; i += SEARCH_CODERS) {
          if (i < n) above[i] = haveAbove ? up(imin(i, nA - 1)) : haveLeft ? lf(0) : 127;
          else if (i < 2 * n) left[i - n] = haveLeft ? lf(imin(i - n, nL - 1)) : haveAbove ? up(0) : 129;
          else above[-1] = left[-1] = haveAbove && haveLeft ? up(-1) : haveAbove ? up(0) : haveLeft ? lf(0) : 128;
        }
      }
      g.sync();
      if (filtered) {
        e.corner = st.pAngle > 90 && st.pAngle < 180 && w + h >= 24;
        e.sa = haveAbove ? pred::edge_strength(w, h, ia.filterType, st.pAngle - 90) : 0;
        e.sl = haveLeft ? pred::edge_strength(w, h, ia.filterType, st.pAngle - 180) : 0;
        e.za = imin(w, maxX - X + 1) + (st.pAngle < 90 ? h : 0) + 1;
        e.zl = imin(h, maxY - Y + 1) + (st.pAngle > 180 ? w : 0) + 1;
      }
      prepare_edges(g, e, above, left, m.edge[2], m.edge[3], w, h);
      const int dcv = mode == DC_PRED ? dc_value(above, left, lw, lh, haveAbove, haveLeft) : 0;
      if (tid == 0) WORK(W_REC_INTRA_PX, w * h);
      const int *wX = sh.smw + w - 4, *wY = sh.smw + h - 4;
      for (int k = tid; k < (w * h) >> 2; k += SEARCH_CODERS) {
        int i = k >> (lw - 2), j0 = (k & ((w >> 2) - 1)) * 4, p[4];
        predict4(mode, e, above, left, wX, wY, w, h, i, j0, dcv, p);
        *(uint32_t *)(sh.px + (y + i) * 64 + x + j0) =
            (uint32_t)(p[0] & 255) | (uint32_t)(p[1] & 255) << 8 | (uint32_t)(p[2] & 255) << 16 | (uint32_t)(p[3] & 255) << 24;
      }
      g.sync();
      int32_t *coefOut = c.coefs + sh.task.coef[0] + (idx << (lw + lh));
      int type = DCT_DCT, eob = 0;
      if (lw > 4 || lh > 4) {
        total += code_large(c, sh, g, txSz, x, y, coefOut, &eob);
      } else {
        if (warp < numCands) eval_candidate(sh, sh.cand[warp], warp, (cands >> (4 * warp)) & 15, txSz, x, y, lane);
        g.sync();
        int bi = 0;
        long long bc = sh.cost[0];
        for (int k = 1; k < numCands; k++)
          if (sh.cost[k] < bc) {
            bc = sh.cost[k];
            bi = k;
          }
        total += bc;
        eob = sh.eob[bi];
        const Cand &cd = sh.cand[bi];
        if (eob) type = (cands >> (4 * bi)) & 15;
        for (int k = tid; k < w * h; k += SEARCH_CODERS) {
          coefOut[k] = cd.q[k];
          if (eob) {
            int i = k >> lw, j = k & (w - 1);
            uint8_t *o = sh.px + (y + i) * 64 + x + j;
            *o = (uint8_t)clip1((int)*o + cd.r[i * CAND_RS + j]);
          }
        }
      }
      if (tid == 0) {
        if (idx < 16) sh.types[idx] = type;
        if (idx == 0) sh.anyNz = 0;
        sh.anyNz |= eob > 0;
        sh.maxW = X + w;
        sh.maxH = Y + h;
      }
      idx++;
      g.sync();
    }
  *nTx = idx;
  return total;
}

__device__ __forceinline__ void set_types(SearchShared &sh, const int *types, int n) {
  for (int k = 0; k < imin(n, 16); k++) {
    int s = 4 * (k & 7);
    int &v = k < 8 ? sh.lo : sh.hi;
    v = (int32_t)(((uint32_t)v & ~(15u << s)) | (uint32_t)types[k] << s);
  }
  if (n > 0) sh.type0 = types[0];
}

__device__ void search_worker(const Ctx &c, SearchShared &sh) {
  const Group<SEARCH_CODERS> g{(int)threadIdx.x, 1};
  const FrameParams *fp = &sh.fpc;
  const int tid = g.tid, fs = fp->stride[0];
  for (;;) {
    record_bar<SEARCH_WORKERS>();
    const int me = sh.task.me;
    if (me < 0) return;
    const PlaneTask &t = sh.task.p[0];
    const int lw = t.geo & 7, w = 1 << lw, h = 1 << ((t.geo >> 3) & 7), wl = lw - 2;
    const uint8_t *sp = c.src + fp->offset[0] + (size_t)t.y * fs + t.x;
    uint8_t *rp = c.rec + fp->offset[0] + (size_t)t.y * fs + t.x;
    BlockInfo *gb = c.blocks + me;
    const bool crosses = t.x + w > fp->mi_cols * 4 || t.y + h > fp->mi_rows * 4;  // transform blocks outside the frame stay as they are
    {  // the block's edges (the corner at [0]), source and record
      const int haveLeft = (t.geo >> 10) & 1, haveAbove = (t.geo >> 11) & 1, ext = imin(w, h);
      const int nA = imin(t.lim & 0xffff, w + ext), nL = imin(t.lim >> 16, h + ext);
      for (int i = tid; i < nA + nL + 2; i += SEARCH_CODERS) {
        if (i <= nA) {
          if (haveAbove && (i > 0 || haveLeft)) sh.above[i] = ldpx(rp - fs + i - 1);
        } else if (haveLeft) {
          int r = i - nA - 1;
          if (r > 0 || haveAbove) sh.left[r] = ldpx(rp + (r - 1) * fs - 1);
        }
      }
      for (int k = tid; k < (w * h) >> 2; k += SEARCH_CODERS) {
        int i = k >> wl, j = 4 * (k & ((1 << wl) - 1));
        *(uint32_t *)(sh.src + i * 64 + j) = __ldg((const uint32_t *)(sp + i * fs + j));
      }
      if (tid == 0) {
        sh.lo = gb->tx_types_lo;
        sh.hi = gb->tx_types_hi;
        sh.type0 = gb->tx_type;
        sh.anyNz = sh.maxW = sh.maxH = 0;
      }
    }
    g.sync();
    const int bs = sh.task.bsize;
    const int maxDepth = fp->tx_mode_select ? imin(MAX_TX_DEPTH, T(Max_Tx_Depth)[bs]) : 0;
    long long best = -1;
    int bestD = 0;
    for (int d = 0; d <= maxDepth; d++) {
      if (crosses) {
        for (int k = tid; k < (w * h) >> 2; k += SEARCH_CODERS) {
          int i = k >> wl, j = 4 * (k & ((1 << wl) - 1));
          *(uint32_t *)(sh.px + i * 64 + j) = __ldcg((const uint32_t *)(rp + i * fs + j));
        }
        g.sync();
      }
      const int txSz = depth_tx_size(bs, d);
      int n = 0;
      long long cst = code_depth(c, sh, g, txSz, &n) + (long long)fp->lambda * 8 * d;
      if (tid == 0) set_types(sh, sh.types, n);
      if (best < 0 || cst < best) {
        best = cst;
        bestD = d;
        if (d < maxDepth) {  // kept for when a later depth has overwritten it
          for (int k = tid; k < (w * h) >> 2; k += SEARCH_CODERS) {
            int i = k >> wl, j = 4 * (k & ((1 << wl) - 1));
            *(uint32_t *)(sh.best + i * 64 + j) = *(const uint32_t *)(sh.px + i * 64 + j);
          }
          const int32_t *cf = c.coefs + sh.task.coef[0];
          for (int k = tid; k < w * h; k += SEARCH_CODERS) sh.bestCoef[k] = __ldcg(cf + k);
          if (tid == 0) {
            for (int k = 0; k < imin(n, 16); k++) sh.bestTypes[k] = sh.types[k];
            sh.bestN = n;
            sh.bestNz = sh.anyNz;
            sh.bestW = sh.maxW;
            sh.bestH = sh.maxH;
          }
        }
      }
      g.sync();
    }
    const uint8_t *px = sh.px;
    if (bestD < maxDepth) {
      // the winner's transform blocks over what the later depths left
      px = sh.best;
      const int txSz = depth_tx_size(bs, bestD), ltx = T(Tx_Width_Log2)[txSz] + T(Tx_Height_Log2)[txSz];
      const int per = imin(32, 1 << T(Tx_Width_Log2)[txSz]) * imin(32, 1 << T(Tx_Height_Log2)[txSz]);
      int32_t *cf = c.coefs + sh.task.coef[0];
      for (int k = tid; k < sh.bestN << ltx; k += SEARCH_CODERS)
        if ((k & ((1 << ltx) - 1)) < per) cf[k] = sh.bestCoef[k];
      if (tid == 0) {
        set_types(sh, sh.bestTypes, sh.bestN);
        sh.anyNz = sh.bestNz;
        sh.maxW = sh.bestW;
        sh.maxH = sh.bestH;
      }
    }
    for (int k = tid; k < (w * h) >> 2; k += SEARCH_CODERS) {
      int i = k >> wl, j = 4 * (k & ((1 << wl) - 1));
      *(uint32_t *)(rp + i * fs + j) = *(const uint32_t *)(px + i * 64 + j);
    }
    if (tid == 0) {
      gb->tx_depth = bestD;
      gb->interp_filter = sh.task.interp;
      gb->tx_type = sh.type0;
      gb->tx_types_lo = sh.lo;
      gb->tx_types_hi = sh.hi;
      gb->eob[0] = sh.anyNz;
      c.tasks[me].maxLumaW = sh.maxW;  // the last transform block coded: CfL's limits
      c.tasks[me].maxLumaH = sh.maxH;
      *(volatile int *)&sh.coded = 1;
    }
    coded_bar<SEARCH_WORKERS>();
  }
}

// Every intra block of the frame, one persistent launch: even CTAs code luma,
// odd ones chroma.
template <bool SEARCH>
__global__ void __launch_bounds__(SEARCH ? SEARCH_WORKERS : WORKER_THREADS, SEARCH ? 2 : 4) k_recon_blocks(Ctx c) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int total = c.counters[CNT_TOTAL], kind = blockIdx.x & 1, tid = threadIdx.x;
  if ((int)(blockIdx.x >> 1) >= imax(MIN_WORKERS, total / BLOCKS_PER_WORKER)) return;
  if (SEARCH && kind == 0) {
    SearchShared &sh = *(SearchShared *)smem_raw;
    load_intra_shared(c, sh);
    if (tid >= SEARCH_CODERS) feed<SEARCH_WORKERS>(c, sh, 0, total);
    else search_worker(c, sh);
    return;
  }
  IntraShared &sh = *(IntraShared *)smem_raw;
  load_intra_shared(c, sh);
  if (tid >= WORKER_THREADS) return;
  if (tid >= CODERS) feed<WORKER_THREADS>(c, sh, kind, total);
  else if (kind == 0) luma_worker(c, sh);
  else chroma_worker(c, sh);
}

// Lossless frames: the reconstruction is the source (the Walsh-Hadamard
// transform and its levels are exact), so the samples an intra block reads
// from its coded neighbours are the source's, and no block waits for another.
// One CTA per block slot; the edges come from the source frame, equal to the
// reconstruction over the coded area that edge limits stay in.
__global__ void __launch_bounds__(INTRA_THREADS) k_recon_lossless(Ctx cg) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem &sm = *(Smem *)smem_raw;
  const int me = blockIdx.x, sb = me / MAX_BLOCKS_PER_SB, tid = threadIdx.x;
  if (me % MAX_BLOCKS_PER_SB >= cg.sbs[sb].num_blocks || cg.blocks[me].is_inter) return;
  if (me == cg.hold) {  // never released (Ctx::hold): its wait gives up, like a dependency wait of k_recon_blocks
    if (tid == 0) {
      volatile int *abort = cg.status + 1;
      int spins = 0;
      while (!*abort && spins++ <= cg.spin_limit) __nanosleep(32);
      if (!*abort) {
        atomicExch(cg.status, 1);
        atomicExch(cg.status + 1, 1);
      }
    }
    return;
  }
  const Ctx c = load_shared(cg, sm);
  const FrameParams *fp = c.fp;
  const int r0 = (sb / fp->sb_cols) * 16, c0 = (sb % fp->sb_cols) * 16;
  if (tid < (int)(sizeof(BlockInfo) / 4)) ((int *)&sm.blk)[tid] = ((const int *)(c.blocks + me))[tid];
  if (tid == 32) {
    sm.r0 = r0;
    sm.c0 = c0;
    sm.maxLumaW = sm.maxLumaH = 0;
  }
  __syncthreads();
  int cb = 0;
  for (int p = 0; p < 2; p++)
    for (int k = 0; k < 2; k++) cb |= corner_decoded(fp, c.blk_at, sm.blk, me, r0, c0, p, k) << (2 * p + k);
  stage_block(c, sm, c.src, cb);
  for (int p = 0; p < 3; p++) code_plane<false>(c, sm, p, TX_4X4);
  unstage_intra(c, sm);
  if (tid == 0) {
    sm.blk.tx_depth = 0;
    sm.blk.interp_filter &= 0x30;
    c.blocks[me] = sm.blk;
  }
}

constexpr size_t SMEM_SINGLE = sizeof(IntraShared);
constexpr size_t SMEM_SEARCH = sizeof(SearchShared) > sizeof(IntraShared) ? sizeof(SearchShared) : sizeof(IntraShared);
constexpr int SINGLE_THREADS = WORKER_THREADS, SEARCH_THREADS = SEARCH_WORKERS;

}  // namespace rec
