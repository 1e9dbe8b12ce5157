// In-loop filters: loop-filter info, deblocking (spec 7.14), CDEF
// (spec 7.15) with per-superblock preset selection, loop restoration apply
// (spec 7.17). Reference: src/kernels/k_lf.h, k_cdef.h, k_lr.h, the filter
// stage of src/backend_cpu.c:158-188 and the host helpers build_filter_info
// and cdef_select (src/encoder.c:513-563).
//
// B200 mapping. Deblocking: one thread per (plane, edge, sample line); the
// spec makes the edges of one pass independent (a filter never reaches the
// samples another edge of the same pass modifies), so a pass is one launch.
// CDEF: a warp per 8x8 block over a shared tile of 8 blocks: the direction
// search accumulates its partial sums in shared memory, then a lane filters
// two luma samples and a chroma sample for every preset. Preset selection: one CTA
// per superblock reduces the SSE of every preset and copies the winner into
// the reconstruction. Loop restoration: one thread per 4x4 block.
#pragma once

#include "common.cuh"

namespace flt {

// ---- loop filter info (encoder.c:513-526) --------------------------------------------
// A CTA per superblock whose blocks go at once, 4 to 32 lanes each over a
// block's units, the more the fewer blocks there are. (A thread per block wrote
// a 64x64 block's 256 units one after another, 24 us for any frame that has
// one; a warp per block took the 64 blocks of a divided superblock in 8 turns,
// 11.1 us on a 352x288 key frame of small blocks against a thread's 8.8, 14.9
// on a 3840x2160 one. This takes 7.5 and 9.2, and 7 for large blocks.)
constexpr int INFO_THREADS = 4 * MAX_BLOCKS_PER_SB;
__global__ void __launch_bounds__(INFO_THREADS) k_filter_info(const FrameParams *fp, const BlockInfo *blocks, const SbInfo *sbs,
                                                              uint8_t *info) {
  const int sb = blockIdx.x, n = sbs[sb].num_blocks, lg = lanes_per_block(n), lane = threadIdx.x & ((1 << lg) - 1);
  const int rows = fp->mi_rows, cols = fp->mi_cols;
  for (int k = threadIdx.x >> lg; k < n; k += INFO_THREADS >> lg) {
    const BlockInfo *b = &blocks[sbs[sb].first_block + k];
    int skip = b->eob[0] == 0 && b->eob[1] == 0 && b->eob[2] == 0;
    int lw = 31 - __clz(T(Num_4x4_Blocks_Wide)[b->bsize]), bh4 = T(Num_4x4_Blocks_High)[b->bsize];
    uint8_t v = (uint8_t)(b->bsize | (skip << 5) | (b->tx_depth << 6));
    for (int i = lane; i < bh4 << lw; i += 1 << lg) {
      int y = b->mi_row + (i >> lw), x = b->mi_col + (i & ((1 << lw) - 1));
      if (y < rows && x < cols) info[y * cols + x] = v;
    }
  }
}

// ---- deblocking (k_lf.h:13-136) ---------------------------------------------------
HD int lf_tx_size(int info, int plane) {
  return plane == 0 ? depth_tx_size(info & 31, (info >> 6) & 3) : uv_tx_size(info & 31, 1, 1);
}

__device__ void lf_sample(uint8_t *px, int pitch, int plane, int lvl, int sharp, int filterSize) {
  int shift = sharp > 4 ? 2 : (sharp > 0 ? 1 : 0);
  int limit = sharp > 0 ? clip3(1, 9 - sharp, lvl >> shift) : imax(1, lvl >> shift);
  int blimit = 2 * (lvl + 2) + limit;
  int thresh = lvl >> 4;
#define S(k) ((int)px[(k) * pitch])
  int q0 = S(0), q1 = S(1), p0 = S(-1), p1 = S(-2);
  int filterLen = filterSize == 4 ? 4 : (plane != 0 ? 6 : (filterSize == 8 ? 8 : 16));
  int q2 = 0, q3 = 0, p2 = 0, p3 = 0;
  if (filterLen >= 6 || filterSize >= 8) {
    q2 = S(2);
    p2 = S(-3);
  }
  if (filterLen >= 8) {
    q3 = S(3);
    p3 = S(-4);
  }
  int hevMask = (iabs(p1 - p0) > thresh) || (iabs(q1 - q0) > thresh);
  int mask = 0;
  mask |= iabs(p1 - p0) > limit;
  mask |= iabs(q1 - q0) > limit;
  mask |= iabs(p0 - q0) * 2 + iabs(p1 - q1) / 2 > blimit;
  if (filterLen >= 6) {
    mask |= iabs(p2 - p1) > limit;
    mask |= iabs(q2 - q1) > limit;
  }
  if (filterLen >= 8) {
    mask |= iabs(p3 - p2) > limit;
    mask |= iabs(q3 - q2) > limit;
  }
  if (mask) return;
  int flatMask = 0, flatMask2 = 0;
  if (filterSize >= 8) {
    int m = 0;
    m |= iabs(p1 - p0) > 1;
    m |= iabs(q1 - q0) > 1;
    m |= iabs(p2 - p0) > 1;
    m |= iabs(q2 - q0) > 1;
    if (filterLen >= 8) {
      m |= iabs(p3 - p0) > 1;
      m |= iabs(q3 - q0) > 1;
    }
    flatMask = m == 0;
  }
  if (filterSize >= 16) {
    int q4 = S(4), q5 = S(5), q6 = S(6), p4 = S(-5), p5 = S(-6), p6 = S(-7);
    int m = 0;
    m |= iabs(p6 - p0) > 1;
    m |= iabs(q6 - q0) > 1;
    m |= iabs(p5 - p0) > 1;
    m |= iabs(q5 - q0) > 1;
    m |= iabs(p4 - p0) > 1;
    m |= iabs(q4 - q0) > 1;
    flatMask2 = m == 0;
  }
  if (filterSize == 4 || !flatMask) {
    int ps1 = p1 - 128, ps0 = p0 - 128, qs0 = q0 - 128, qs1 = q1 - 128;
    int filter = hevMask ? clip3(-128, 127, ps1 - qs1) : 0;
    filter = clip3(-128, 127, filter + 3 * (qs0 - ps0));
    int filter1 = clip3(-128, 127, filter + 4) >> 3;
    int filter2 = clip3(-128, 127, filter + 3) >> 3;
    px[0] = (uint8_t)(clip3(-128, 127, qs0 - filter1) + 128);
    px[-pitch] = (uint8_t)(clip3(-128, 127, ps0 + filter2) + 128);
    if (!hevMask) {
      filter = round2(filter1, 1);
      px[pitch] = (uint8_t)(clip3(-128, 127, qs1 - filter) + 128);
      px[-2 * pitch] = (uint8_t)(clip3(-128, 127, ps1 + filter) + 128);
    }
  } else {
    int log2Size = (filterSize == 8 || !flatMask2) ? 3 : 4;
    int n = log2Size == 4 ? 6 : (plane == 0 ? 3 : 2);
    int n2 = (log2Size == 3 && plane == 0) ? 0 : 1;
    int v[14];
    for (int k = -(n + 1); k <= n; k++) v[k + 7] = S(k);
    int F[12];
    for (int i = -n; i < n; i++) {
      int t = 0;
      for (int j = -n; j <= n; j++) {
        int p = clip3(-(n + 1), n, i + j);
        int tap = iabs(j) <= n2 ? 2 : 1;
        t += v[p + 7] * tap;
      }
      F[i + n] = round2(t, log2Size);
    }
    for (int i = -n; i < n; i++) px[i * pitch] = (uint8_t)F[i + n];
  }
#undef S
}

// One pass (0: vertical edges, 1: horizontal edges); thread per (edge position
// k, sample i) of a line of units, blockIdx.y the line, blockIdx.z the plane
// (chroma: every second line and position). The thread index used to be
// divided into them in 64 bits.
constexpr int LF_THREADS = 128;
__global__ void __launch_bounds__(LF_THREADS) k_deblock(const FrameParams *fp, uint8_t *rec, const uint8_t *miSizes, int pass) {
  const int plane = blockIdx.z, sub = plane > 0;
  const int lines = pass == 0 ? fp->mi_rows : fp->mi_cols, n = pass == 0 ? fp->mi_cols : fp->mi_rows;
  const int g = blockIdx.x * LF_THREADS + threadIdx.x, i = g & 3, k = (g >> 2) << sub, line = blockIdx.y << sub;
  if (line >= lines || k >= n) return;
  int lvl = clip3(0, MAX_LOOP_FILTER, fp->lf_level[plane == 0 ? pass : plane + 1]);
  if (lvl == 0) return;
  int stride = fp->stride[plane];
  uint8_t *base = rec + fp->offset[plane];
  int dx = pass == 0, dy = pass == 1;
  int row0 = pass == 0 ? line : k, col0 = pass == 0 ? k : line;
  int x = col0 * MI_SIZE, y = row0 * MI_SIZE;
  int row = row0 | sub, col = col0 | sub;
  if (x >= fp->frame_w || y >= fp->frame_h) return;
  if (pass == 0 && x == 0) return;
  if (pass == 1 && y == 0) return;
  int xP = x >> sub, yP = y >> sub;
  int prevRow = row - (dy << sub), prevCol = col - (dx << sub);
  int txSz = lf_tx_size(miSizes[row * fp->mi_cols + col], plane);
  int prevTxSz = lf_tx_size(miSizes[prevRow * fp->mi_cols + prevCol], plane);
  int isTxEdge = pass == 0 ? (xP % T(Tx_Width)[txSz]) == 0 : (yP % T(Tx_Height)[txSz]) == 0;
  if (!isTxEdge) return;
  int baseSize = pass == 0 ? imin(T(Tx_Width)[prevTxSz], T(Tx_Width)[txSz]) : imin(T(Tx_Height)[prevTxSz], T(Tx_Height)[txSz]);
  int filterSize = plane == 0 ? imin(16, baseSize) : imin(8, baseSize);
  int sx = xP + dy * i, sy = yP + dx * i;
  WORK(W_LF_TAPS, filterSize == 4 ? 4 : (plane != 0 ? 6 : (filterSize == 8 ? 8 : 16)));  // the line's filter length
  lf_sample(base + sy * stride + sx, pass == 0 ? 1 : stride, plane, lvl, fp->lf_sharpness, filterSize);
}

// ---- CDEF (k_cdef.h:9-150) ------------------------------------------------------------
// A CTA of 8 warps takes 8 neighbouring 8x8 blocks, a warp each. Their samples
// and the 2 around them lie in shared memory as 16-bit values, CDEF_FAR where
// CdefAvailable is 0 (outside the frame's units): such a tap's constrained
// difference is 0 and it takes no part in the clamp, so no tap needs a
// position check, and the sums are those of k_cdef.h's taps. (A sample a
// thread with checked taps from the frame, and a constrain( ) that looked for
// its threshold's logarithm bit by bit at every tap: 117 us for a 1080p frame
// and one filtering preset.)
constexpr int CDEF_THREADS = 256, CDEF_YP = 72, CDEF_CP = 40;
constexpr int CDEF_FAR = 30000;
struct CdefMem {
  uint16_t y[12 * CDEF_YP];      // rows -2 .. 9, columns -4 .. 67
  uint16_t c[2][8 * CDEF_CP];    // rows -2 .. 5, columns -4 .. 35
  int partial[CDEF_THREADS / 32][8][16];
  int weight[8][16];             // of each direction's lines in its cost
};

// Filtered value of the sample at t (row pitch P) with primary strength pri
// (damping shift priSh) along d0, secondary sec along the directions beside.
template <int P>
__device__ __forceinline__ int cdef_sample(const uint16_t *t, int dir, int pri, int priSh, int sec, int secSh, int tapSet) {
  const int x = *t;
  int sum = 0, mx = x, mn = x;
#pragma unroll
  for (int part = 0; part < 3; part++) {
    const int d = part == 0 ? dir : (dir + (part == 1 ? -2 : 2)) & 7, thr = part == 0 ? pri : sec, sh = part == 0 ? priSh : secSh;
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int o = T(Cdef_Directions)[d][k][0] * P + T(Cdef_Directions)[d][k][1];
      const int w = part == 0 ? T(Cdef_Pri_Taps)[tapSet][k] : T(Cdef_Sec_Taps)[tapSet][k];
#pragma unroll
      for (int sg = 0; sg < 2; sg++) {
        const int p = t[sg ? o : -o], df = p - x, ad = iabs(df);
        const int r = imin(ad, imax(0, thr - (ad >> sh)));
        sum += w * (df < 0 ? -r : r);
        mx = imax(mx, p == CDEF_FAR ? x : p);
        mn = imin(mn, p);
      }
    }
  }
  return clip3(mn, mx, x + ((8 + sum - (sum < 0)) >> 4));
}
__device__ __forceinline__ int cdef_shift(int strength, int damping) {
  return strength ? imax(0, damping - (31 - __clz(strength))) : 0;
}

__global__ void __launch_bounds__(CDEF_THREADS) k_cdef(const FrameParams *fp, const uint8_t *cur, uint8_t *out, long long frameBytes,
                                                      const uint8_t *info, int npresets) {
  __shared__ CdefMem m;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r = blockIdx.y * 2, c0 = blockIdx.x * 16, cols = fp->mi_cols, rows = fp->mi_rows;
  // samples, a word of 4 a thread: the frame's units cover whole words
  if (tid < 12 * (CDEF_YP / 4)) {
    int i = tid / (CDEF_YP / 4), j = tid - i * (CDEF_YP / 4), y = r * 4 - 2 + i, x = c0 * 4 - 4 + 4 * j;
    bool in = y >= 0 && y < rows * 4 && x >= 0 && x < cols * 4;
    uint32_t v = in ? *(const uint32_t *)(cur + fp->offset[0] + y * fp->stride[0] + x) : 0;
    for (int e = 0; e < 4; e++) m.y[i * CDEF_YP + 4 * j + e] = in ? (v >> (8 * e)) & 255 : CDEF_FAR;
  }
  if (tid < 2 * 8 * (CDEF_CP / 4)) {
    int p = tid / (8 * (CDEF_CP / 4)), q = tid - p * (8 * (CDEF_CP / 4)), i = q / (CDEF_CP / 4), j = q - i * (CDEF_CP / 4);
    int y = r * 2 - 2 + i, x = c0 * 2 - 4 + 4 * j;
    bool in = y >= 0 && y < rows * 2 && x >= 0 && x < cols * 2;
    uint32_t v = in ? *(const uint32_t *)(cur + fp->offset[1 + p] + y * fp->stride[1 + p] + x) : 0;
    for (int e = 0; e < 4; e++) m.c[p][i * CDEF_CP + 4 * j + e] = in ? (v >> (8 * e)) & 255 : CDEF_FAR;
  }
  if (tid < 128) {
    int d = tid >> 4, k = tid & 15, w = 0;
    if (d == 2 || d == 6) w = k < 8 ? 8 : 0;
    else if (d == 0 || d == 4) w = k < 8 ? k + 1 : k < 15 ? 15 - k : 0;
    else w = k < 3 ? 2 * k + 2 : k < 8 ? 8 : k < 11 ? 2 * (10 - k) + 2 : 0;
    m.weight[d][k] = w ? T(Div_Table)[w] : 0;
  }
  __syncthreads();
  const int c = c0 + 2 * warp;
  if (c >= cols) return;
  const int skip = (info[r * cols + c] >> 5) & 1;
  const uint16_t *ty = m.y + 2 * CDEF_YP + 4 + 8 * warp;
  // this lane's luma samples (row i, columns j, j + 1) and chroma sample
  const int i = lane >> 2, j = (lane & 3) * 2, cp = lane >> 4, ci = (lane >> 2) & 3, cj = lane & 3;
  int dir = 0, var = 0;
  if (!skip) {
    if (lane == 0) WORK(W_CDEF_TAPS, 64 * 8);  // direction search: 64 samples into 8 projections
    int(*pt)[16] = m.partial[warp];
    for (int k = lane; k < 128; k += 32) pt[k >> 4][k & 15] = 0;
    __syncwarp();
    for (int e = 0; e < 2; e++) {
      int jj = j + e, x = (int)ty[i * CDEF_YP + jj] - 128;
      atomicAdd(&pt[0][i + jj], x);
      atomicAdd(&pt[1][i + jj / 2], x);
      atomicAdd(&pt[2][i], x);
      atomicAdd(&pt[3][3 + i - jj / 2], x);
      atomicAdd(&pt[4][7 + i - jj], x);
      atomicAdd(&pt[5][3 - i / 2 + jj], x);
      atomicAdd(&pt[6][jj], x);
      atomicAdd(&pt[7][i / 2 + jj], x);
    }
    __syncwarp();
    // four lanes a direction
    const int d = lane >> 2;
    int cost = 0;
    for (int k = lane & 3; k < 15; k += 4) cost += pt[d][k] * pt[d][k] * m.weight[d][k];
    cost += __shfl_xor_sync(0xffffffffu, cost, 1);
    cost += __shfl_xor_sync(0xffffffffu, cost, 2);
    int best = __reduce_max_sync(0xffffffffu, cost);
    dir = (__ffs(__ballot_sync(0xffffffffu, cost == best)) - 1) >> 2;  // the first greatest
    var = (best - __shfl_sync(0xffffffffu, cost, ((dir + 4) & 7) * 4)) >> 10;
  }
  const size_t yo = fp->offset[0] + (size_t)(r * 4 + i) * fp->stride[0] + c * 4 + j;
  const size_t co = fp->offset[1 + cp] + (size_t)(r * 2 + ci) * fp->stride[1 + cp] + c * 2 + cj;
  const uint16_t *sy = ty + i * CDEF_YP + j, *sc = m.c[cp] + (2 + ci) * CDEF_CP + 4 + 4 * warp + cj;
  for (int idx = 0; idx < npresets; idx++) {
    uint8_t *o = out + (long long)idx * frameBytes;
    const int priStr = fp->cdef_y_pri[idx], secStr = fp->cdef_y_sec[idx], uvPri = fp->cdef_uv_pri[idx], uvSec = fp->cdef_uv_sec[idx];
    int a = sy[0], b = sy[1], v = sc[0];
    if (!(skip || (priStr == 0 && secStr == 0 && uvPri == 0 && uvSec == 0))) {
      if (lane == 0) WORK(W_CDEF_TAPS, (64 + 32) * 12);  // 12 taps per filtered sample
      const int varStr = (var >> 6) ? imin(31 - __clz(var >> 6), 12) : 0, pri = var ? (priStr * (4 + varStr) + 8) >> 4 : 0;
      const int yd = priStr == 0 ? 0 : dir, cd = uvPri == 0 ? 0 : T(Cdef_Uv_Dir)[1][1][dir], damp = fp->cdef_damping;
      const int ps = cdef_shift(pri, damp), ss = cdef_shift(secStr, damp);
      a = cdef_sample<CDEF_YP>(sy, yd, pri, ps, secStr, ss, pri & 1);
      b = cdef_sample<CDEF_YP>(sy + 1, yd, pri, ps, secStr, ss, pri & 1);
      v = cdef_sample<CDEF_CP>(sc, cd, uvPri, cdef_shift(uvPri, damp - 1), uvSec, cdef_shift(uvSec, damp - 1), uvPri & 1);
    }
    *(uint16_t *)(o + yo) = (uint16_t)(a | b << 8);
    o[co] = (uint8_t)v;
  }
}

// Per superblock: SSE of every preset against the source (real frame area),
// first minimum, copy of the winner into rec (mi-aligned area)
// (cdef_select, encoder.c:530-563).
__global__ void __launch_bounds__(256) k_cdef_select(const FrameParams *fp, const uint8_t *src, const uint8_t *cdefbuf,
                                                     long long frameBytes, uint8_t *rec, int8_t *choice, int npresets) {
  __shared__ long long red[8][4];
  __shared__ int s_best;
  int sb = blockIdx.x;
  int sr = sb / fp->sb_cols, sc = sb % fp->sb_cols;
  int tid = threadIdx.x;
  long long sse[4] = {0, 0, 0, 0};
  for (int p = 0; p < 3; p++) {
    const int sub = p > 0, ln = 6 - sub, n = 64 >> sub;
    const int pw = p ? (fp->frame_w + 1) >> 1 : fp->frame_w, ph = p ? (fp->frame_h + 1) >> 1 : fp->frame_h;
    int part[4] = {0, 0, 0, 0};  // at most 16 samples of 255^2
    for (int k = tid; k < n * n / 4; k += 256) {
      const int y = sr * n + (k >> (ln - 2)), x = sc * n + (k & (n / 4 - 1)) * 4;
      if (y >= ph || x >= pw) continue;
      const size_t o = fp->offset[p] + (size_t)y * fp->stride[p] + x;
      const uint32_t keep = pw - x >= 4 ? 0xffffffffu : (1u << (8 * (pw - x))) - 1;  // samples inside the frame
      const uint32_t s = *(const uint32_t *)(src + o);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if (q >= npresets) break;
        uint32_t d = __vabsdiffu4(*(const uint32_t *)(cdefbuf + (size_t)q * frameBytes + o), s) & keep;
        part[q] = (int)__dp4a(d, d, (unsigned)part[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) sse[q] += part[q];
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    if (q >= npresets) break;
    long long v = sse[q];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if ((tid & 31) == 0) red[tid >> 5][q] = v;
  }
  __syncthreads();
  if (tid == 0) {
    long long best = -1;
    int bestK = 0;
    for (int q = 0; q < npresets; q++) {
      long long s = 0;
      for (int w = 0; w < 8; w++) s += red[w][q];
      if (best < 0 || s < best) {
        best = s;
        bestK = q;
      }
    }
    s_best = bestK;
    choice[sb] = (int8_t)bestK;
  }
  __syncthreads();
  const uint8_t *out = cdefbuf + (size_t)s_best * frameBytes;
  for (int p = 0; p < 3; p++) {
    const int sub = p > 0, ln = 6 - sub, n = 64 >> sub;
    const int mw = (fp->mi_cols * 4) >> sub, mh = (fp->mi_rows * 4) >> sub;  // multiples of 4
    for (int k = tid; k < n * n / 4; k += 256) {
      const int y = sr * n + (k >> (ln - 2)), x = sc * n + (k & (n / 4 - 1)) * 4;
      if (y >= mh || x >= mw) continue;
      const size_t o = fp->offset[p] + (size_t)y * fp->stride[p] + x;
      *(uint32_t *)(rec + o) = *(const uint32_t *)(out + o);
    }
  }
}

// ---- loop restoration apply (k_lr.h:28-202) ----------------------------------------------
struct LrBlock {
  int x, y, w, h;
  int stripeStart, stripeEnd;
  int planeEndX, planeEndY;
  int unitRow, unitCol;
};

HD int lr_block_setup(const FrameParams *fp, int plane, int row, int col, LrBlock *lb) {
  int sub = plane > 0;
  int lumaY = row * MI_SIZE;
  int stripeNum = (lumaY + 8) / 64;
  lb->stripeStart = (-8 + stripeNum * 64) >> sub;
  lb->stripeEnd = lb->stripeStart + (64 >> sub) - 1;
  int unitSize = fp->lr_unit_size[plane];
  lb->unitRow = imin(fp->lr_unit_rows[plane] - 1, ((row * MI_SIZE + 8) >> sub) / unitSize);
  lb->unitCol = imin(fp->lr_unit_cols[plane] - 1, ((col * MI_SIZE) >> sub) / unitSize);
  lb->planeEndX = ((fp->frame_w + sub) >> sub) - 1;
  lb->planeEndY = ((fp->frame_h + sub) >> sub) - 1;
  lb->x = (col * MI_SIZE) >> sub;
  lb->y = (row * MI_SIZE) >> sub;
  lb->w = imin(MI_SIZE >> sub, lb->planeEndX - lb->x + 1);
  lb->h = imin(MI_SIZE >> sub, lb->planeEndY - lb->y + 1);
  return lb->w > 0 && lb->h > 0;
}

// get_source_sample( ) (spec 7.17.6)
HD int lr_src(const FrameParams *fp, int plane, const LrBlock *lb, const uint8_t *cdef, const uint8_t *dbk, int x, int y) {
  x = imax(0, imin(lb->planeEndX, x));
  y = imax(0, imin(lb->planeEndY, y));
  int stride = fp->stride[plane];
  if (y < lb->stripeStart) {
    y = imax(lb->stripeStart - 2, y);
    return dbk[fp->offset[plane] + y * stride + x];
  } else if (y > lb->stripeEnd) {
    y = imin(lb->stripeEnd + 2, y);
    return dbk[fp->offset[plane] + y * stride + x];
  }
  return cdef[fp->offset[plane] + y * stride + x];
}

// The samples the loop-restoration filters read, get_source_sample( ) for the
// filter taps and the CDEF output at the block's own positions, and the picture
// they write. (The parameter search has its own filters, over a unit's samples
// in shared memory.)
struct LrFrame {
  const FrameParams *fp;
  int plane;
  const uint8_t *cdef, *dbk;
  uint8_t *out;
  HD int tap(const LrBlock *lb, int x, int y) const { return lr_src(fp, plane, lb, cdef, dbk, x, y); }
  HD int own(int x, int y) const { return cdef[fp->offset[plane] + y * fp->stride[plane] + x]; }
  HD void store(int x, int y, int v) const { out[fp->offset[plane] + y * fp->stride[plane] + x] = (uint8_t)v; }
};

// Wiener filter (spec 7.17.4, 8-bit rounding).
HD void lr_wiener(const LrBlock *lb, const LrFrame &in, const LrUnit *u) {
  int vf[7], hf[7];
  vf[3] = 128;
  hf[3] = 128;
  for (int i = 0; i < 3; i++) {
    vf[i] = vf[6 - i] = u->wiener[0][i];
    vf[3] -= 2 * u->wiener[0][i];
    hf[i] = hf[6 - i] = u->wiener[1][i];
    hf[3] -= 2 * u->wiener[1][i];
  }
  const int round0 = 3, round1 = 11;
  int offset = 1 << (8 + FILTER_BITS - round0 - 1);
  int limit = (1 << (8 + 1 + FILTER_BITS - round0)) - 1;
  int inter[10][4];
  for (int r = 0; r < lb->h + 6; r++)
    for (int c = 0; c < lb->w; c++) {
      int s = 0;
      for (int t = 0; t < 7; t++) s += hf[t] * in.tap(lb, lb->x + c + t - 3, lb->y + r - 3);
      inter[r][c] = clip3(-offset, limit - offset, round2(s, round0));
    }
  for (int r = 0; r < lb->h; r++)
    for (int c = 0; c < lb->w; c++) {
      int s = 0;
      for (int t = 0; t < 7; t++) s += vf[t] * inter[r + t][c];
      in.store(lb->x + c, lb->y + r, clip3(0, 255, round2(s, round1)));
    }
}

// Box filter (spec 7.17.3); F gets w x h values (row stride 4).
HD void lr_box(const LrBlock *lb, const LrFrame &in, int set, int pass, int *F) {
  int r = T(Sgr_Params)[set][pass * 2 + 0];
  if (r == 0) return;
  int eps = T(Sgr_Params)[set][pass * 2 + 1];
  int A[6][6], Bv[6][6];
  int n = (2 * r + 1) * (2 * r + 1);
  int n2e = n * n * eps;
  int s = ((1 << SGRPROJ_MTABLE_BITS) + n2e / 2) / n2e;
  int oneOverN = ((1 << SGRPROJ_RECIP_BITS) + (n / 2)) / n;
  for (int i = -1; i < lb->h + 1; i++)
    for (int j = -1; j < lb->w + 1; j++) {
      long long a = 0, b = 0;
      for (int dy = -r; dy <= r; dy++)
        for (int dx = -r; dx <= r; dx++) {
          long long c = in.tap(lb, lb->x + j + dx, lb->y + i + dy);
          a += c * c;
          b += c;
        }
      long long d = b;
      long long p = a * n - d * d;
      if (p < 0) p = 0;
      long long z = (p * s + (1LL << (SGRPROJ_MTABLE_BITS - 1))) >> SGRPROJ_MTABLE_BITS;
      long long a2;
      if (z >= 255) a2 = 256;
      else if (z == 0) a2 = 1;
      else a2 = ((z << SGRPROJ_SGR_BITS) + (z / 2)) / (z + 1);
      long long b2 = ((1LL << SGRPROJ_SGR_BITS) - a2) * b * oneOverN;
      A[i + 1][j + 1] = (int)a2;
      Bv[i + 1][j + 1] = (int)((b2 + (1LL << (SGRPROJ_RECIP_BITS - 1))) >> SGRPROJ_RECIP_BITS);
    }
  for (int i = 0; i < lb->h; i++) {
    int shift = 5;
    if (pass == 0 && (i & 1)) shift = 4;
    for (int j = 0; j < lb->w; j++) {
      long long a = 0, b = 0;
      for (int dy = -1; dy <= 1; dy++)
        for (int dx = -1; dx <= 1; dx++) {
          int weight;
          if (pass == 0) weight = ((i + dy) & 1) ? (dx == 0 ? 6 : 5) : 0;
          else weight = (dx == 0 || dy == 0) ? 4 : 3;
          a += weight * A[i + dy + 1][j + dx + 1];
          b += weight * Bv[i + dy + 1][j + dx + 1];
        }
      long long v = a * in.own(lb->x + j, lb->y + i) + b;
      int sh = SGRPROJ_SGR_BITS + shift - SGRPROJ_RST_BITS;
      F[i * 4 + j] = (int)((v + (1LL << (sh - 1))) >> sh);
    }
  }
}

// Self-guided filter (spec 7.17.2): the box filters' outputs projected.
HD void lr_sgr(const LrBlock *lb, const LrFrame &in, const LrUnit *u) {
  int flt0[16], flt1[16];
  lr_box(lb, in, u->set, 0, flt0);
  lr_box(lb, in, u->set, 1, flt1);
  int w0 = u->xqd[0], w1 = u->xqd[1];
  int w2 = (1 << SGRPROJ_PRJ_BITS) - w0 - w1;
  int r0 = T(Sgr_Params)[u->set][0], r1 = T(Sgr_Params)[u->set][2];
  for (int i = 0; i < lb->h; i++)
    for (int j = 0; j < lb->w; j++) {
      int uu = in.own(lb->x + j, lb->y + i) << SGRPROJ_RST_BITS;
      int v = w1 * uu;
      v += r0 ? w0 * flt0[i * 4 + j] : w0 * uu;
      v += r1 ? w2 * flt1[i * 4 + j] : w2 * uu;
      in.store(lb->x + j, lb->y + i, clip3(0, 255, round2(v, SGRPROJ_RST_BITS + SGRPROJ_PRJ_BITS)));
    }
}

// Thread per (plane, 4x4 luma block): loop_restore_block( ) with the unit's
// filter, RESTORE_NONE copies the CDEF output.
__global__ void k_lr_apply(const FrameParams *fp, const uint8_t *cdef, const uint8_t *dbk, uint8_t *out,
                           const LrUnit *units) {
  int rows4 = (fp->frame_h + 3) >> 2, cols4 = (fp->frame_w + 3) >> 2, n = rows4 * cols4;
  int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= 3 * n) return;
  int plane = g / n, i = g % n;
  LrBlock lb;
  if (!lr_block_setup(fp, plane, i / cols4, i % cols4, &lb)) return;
  LrUnit u;
  if (fp->lr_type[plane] == RESTORE_NONE) u.type = RESTORE_NONE;
  else u = units[fp->lr_unit_off[plane] + lb.unitRow * fp->lr_unit_cols[plane] + lb.unitCol];
  WORK(W_LR_TAPS, lb.w * lb.h * (u.type == RESTORE_WIENER ? 14 : u.type == RESTORE_SGRPROJ ? 34 : 0));
  const LrFrame in{fp, plane, cdef, dbk, out};
  if (u.type == RESTORE_WIENER) {
    lr_wiener(&lb, in, &u);
  } else if (u.type == RESTORE_SGRPROJ) {
    lr_sgr(&lb, in, &u);
  } else {
    int stride = fp->stride[plane];
    for (int y = 0; y < lb.h; y++)
      for (int x = 0; x < lb.w; x++) {
        int o = fp->offset[plane] + (lb.y + y) * stride + lb.x + x;
        out[o] = cdef[o];
      }
  }
}

}  // namespace flt
