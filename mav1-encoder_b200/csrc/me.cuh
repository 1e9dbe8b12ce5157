// Hierarchical motion search (reference src/kernels/k_me.h, driven by
// src/backend_cpu.c:23-56).
//
// Per node (64x64 .. 8x8 square of a superblock) and reference: an ordered
// list of full-pel candidates (level 0: a coarse grid, optionally on the
// 4x4-decimated planes, then refinement stages), the first minimum of
// SAD + ac_q * bits / 64, then half- and quarter-pel refinement by the first
// minimum of the 4x4-SATD over the node. The levels depend on each other
// (children search around the parent's vector) and run as separate launches.
//
// B200 mapping: a kernel per level and sub-pel mode (k_me_level). A node and
// reference is searched by half a warp (8x8), a warp, or a CTA (64x64, and 32x32
// without quarter-pel planes). Half a warp's and a warp's lanes take
// candidates (SAD rows on packed bytes with __vsadu4; interior candidates read
// unaligned words through funnel shifts); a CTA's warps take candidates in
// turn, a warp's lanes splitting one's byte pairs; the refinement of +-2
// samples reads a window of 5 rows of 3 words for all its 25 candidates. The
// 64-bit key (cost << 32 | index) is reduced to its minimum, which is exactly
// the serial first minimum. Sub-pel candidates x 4x4 units are spread over the
// group. Quarter-pel planes (16 per reference, EIGHTTAP, the T_ME_HPEL mode)
// are built once per reference picture by their own kernel.
#pragma once

#include "common.cuh"
#include "pred.cuh"

namespace me {

struct Frame {
  const FrameParams *fp;   // device copy
  const uint8_t *src;      // padded source frame
  const uint8_t *ref;      // reference frame (padded layout)
  const uint8_t *qp;       // 16 quarter-pel planes of ref, frame_w x frame_h each
  const uint8_t *dsrc;     // decimated source, dec_w x dec_h
  const uint8_t *dref;     // decimated reference
  int32_t *mv;             // mv field of this reference
  int isGold;
};

HD int dec_w(const FrameParams *fp) { return (fp->frame_w + 3) >> 2; }
HD int dec_h(const FrameParams *fp) { return (fp->frame_h + 3) >> 2; }

// acc + the dot product of four unsigned samples and four signed factors
__device__ __forceinline__ int dp4s(uint32_t px, uint32_t w, int acc) {
  int r;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(px), "r"(w), "r"(acc));
  return r;
}

// ---- quarter-pel and decimated planes -----------------------------------------

// Plane fy * 4 + fx holds the EIGHTTAP prediction of (y + fy / 4, x + fx / 4)
// (k_me.h:289-313): horizontal Round2( ., 3 ), vertical Round2( ., 11 ), Clip1.
// Integer work bounds it, not the 16 W H bytes written: 8 multiply-adds a
// pass and sample, clip and pack took 115 us for a 3840x2160 picture. So
// - the two outer taps of this filter are zero and every tap is even: half
//   taps fit 8 bits, (2 S + 4) >> 3 = (S + 2) >> 2 and (2 S + 1024) >> 11 =
//   (S + 512) >> 10 exactly, a horizontal sum is 2 byte dot products and a
//   vertical one 3 dot products of a 16-bit row pair, and a full-sample phase
//   is the same code with the tap 64;
// - a thread walks down 4 columns of one horizontal phase with the last rows'
//   sums as pairs in registers: no shared memory, 5 extra rows in QP_ROWS + 5.
// 3840x2160: 115 -> 56 us a picture (2.4 TB/s of writes; a leaf frame 1.47 -> 1.38 ms).
// The four phases of a strip are four warps of one CTA, so the reference rows
// come from L1 for three of them.
constexpr int QP_TW = 128, QP_ROWS = 16, QP_STRIPS = 2, QP_TH = QP_ROWS * QP_STRIPS, QP_THREADS = 128 * QP_STRIPS;
constexpr int QP_FILTERS MAV1T_Subpel_Filters_DIMS = MAV1T_Subpel_Filters;

// Half taps t0 .. t0 + 3 of a quarter-pel phase (those past tap 6 are zero) as bytes.
__host__ __device__ constexpr int qp_half(int phase, int t0) {
  uint32_t w = 0;
  for (int t = 0; t < 4 && t0 + t < 8; t++) w |= (uint32_t)((QP_FILTERS[EIGHTTAP][4 * phase][t0 + t] / 2) & 255) << (8 * t);
  return (int)w;
}
constexpr bool qp_taps_fit() {
  for (int p = 0; p < 4; p++) {
    const auto &f = QP_FILTERS[EIGHTTAP][4 * p];
    if (f[0] || f[7]) return false;
    for (int t = 0; t < 8; t++)
      if (f[t] % 2 || f[t] < -256 || f[t] > 254) return false;
  }
  return true;
}
static_assert(qp_taps_fit(), "the quarter-pel filters have six even taps of at most 9 bits");

__global__ void __launch_bounds__(QP_THREADS, 4) k_qpel_planes(const FrameParams *fp, const uint8_t *ref, uint8_t *qp) {
  const int W = fp->frame_w, H = fp->frame_h, stride = fp->stride[0];
  const int tid = threadIdx.x, fx = (tid >> 5) & 3;
  const int x = blockIdx.x * QP_TW + (tid & 31) * 4, y0 = blockIdx.y * QP_TH + (tid >> 7) * QP_ROWS;
  // taps: the horizontal pass over the strips' rows (4 phases), the vertical pass per output of 16 planes
  if (tid == 0)
    WORK(W_QPEL_TAPS, (QP_ROWS + 5) * QP_STRIPS * QP_TW * 4 * 6 +
                          imin(QP_TH, H - (int)blockIdx.y * QP_TH) * imin(QP_TW, W - (int)blockIdx.x * QP_TW) * 16 * 6);
  if (x >= W || y0 >= H) return;
  constexpr int T0[4] = {qp_half(0, 1), qp_half(1, 1), qp_half(2, 1), qp_half(3, 1)};
  constexpr int T1[4] = {qp_half(0, 5), qp_half(1, 5), qp_half(2, 5), qp_half(3, 5)};
  const int t0 = fx < 2 ? (fx ? T0[1] : T0[0]) : (fx == 2 ? T0[2] : T0[3]);
  const int t1 = fx < 2 ? (fx ? T1[1] : T1[0]) : (fx == 2 ? T1[2] : T1[3]);
  // The columns x - 4 .. x + 7 as three aligned words (strides are multiples
  // of 32 samples); columns outside the picture take its edge sample.
  const uint8_t *col = ref + fp->offset[0] + x;
  const int before = x ? -4 : 0, after = x + 4 < stride ? 4 : 0;
  const uint32_t sel0 = x ? 0x3210 : 0;
  uint32_t sel1 = 0, sel2 = 0;
  for (int j = 0; j < 4; j++) {
    sel1 |= (uint32_t)imin(j, W - 1 - x) << (4 * j);
    sel2 |= (uint32_t)imin(4 + j, W - 1 - x) << (4 * j);
  }
  const size_t n = (size_t)W * H;
  uint8_t *out = qp + fx * n + (size_t)y0 * W + x;
  const bool word = (W & 3) == 0;  // every plane row 4-byte aligned
  int prev[4], pair[5][4];  // the last row's sums; sums of rows r and r + 1 as halves, for the last five r
#pragma unroll
  for (int r = 0; r < QP_ROWS + 5; r++) {
    const uint8_t *row = col + (size_t)clip3(0, H - 1, y0 + r - 2) * stride;
    uint32_t l0 = __ldg((const uint32_t *)(row + before)), l1 = __ldg((const uint32_t *)row),
             l2 = __ldg((const uint32_t *)(row + after));
    uint32_t w0 = __byte_perm(l0, l0, sel0), w1 = __byte_perm(l1, l2, sel1), w2 = __byte_perm(l1, l2, sel2);
    int h[4];
    h[0] = dp4s(__funnelshift_r(w1, w2, 16), t1, dp4s(__funnelshift_r(w0, w1, 16), t0, 2)) >> 2;
    h[1] = dp4s(__funnelshift_r(w1, w2, 24), t1, dp4s(__funnelshift_r(w0, w1, 24), t0, 2)) >> 2;
    h[2] = dp4s(w2, t1, dp4s(w1, t0, 2)) >> 2;
    h[3] = dp4s(w2 >> 8, t1, dp4s(__funnelshift_r(w1, w2, 8), t0, 2)) >> 2;
    for (int k = 0; k < 4; k++) {
      if (r) pair[(r - 1) % 5][k] = (int)__byte_perm((uint32_t)prev[k], (uint32_t)h[k], 0x5410);
      prev[k] = h[k];
    }
    if (r < 5) continue;
    if (y0 + r - 5 >= H) return;
    for (int fy = 0; fy < 4; fy++) {
      int v[4];
      for (int k = 0; k < 4; k++) {
        int s = __dp2a_hi(pair[(r - 3) % 5][k], T0[fy], 512);
        if (fy) s = __dp2a_lo(pair[(r - 1) % 5][k], T1[fy], __dp2a_lo(pair[(r - 5) % 5][k], T0[fy], s));
        v[k] = s >> 10;
      }
      uint8_t *o = out + (size_t)fy * 4 * n;
      if (word) {
        uint32_t hi, packed;  // saturating to 0 .. 255
        asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, 0;" : "=r"(hi) : "r"(v[3]), "r"(v[2]));
        asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(packed) : "r"(v[1]), "r"(v[0]), "r"(hi));
        *(uint32_t *)o = packed;
      } else {
        for (int k = 0; k < 4; k++)
          if (x + k < W) o[k] = (uint8_t)clip1(v[k]);
      }
    }
    out += W;
  }
}

// 4x4 average of the frame, (sum + 8) >> 4 (k_me.h:112-118).
__global__ void k_dec_plane(const FrameParams *fp, const uint8_t *pl, uint8_t *out) {
  int W = dec_w(fp), H = dec_h(fp);
  int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= W || y >= H) return;
  int s = 0;
  for (int i = 0; i < 4; i++)
    for (int j = 0; j < 4; j++)
      s += pl[fp->offset[0] + clip3(0, fp->frame_h - 1, 4 * y + i) * fp->stride[0] + clip3(0, fp->frame_w - 1, 4 * x + j)];
  out[(size_t)y * W + x] = (uint8_t)((s + 8) >> 4);
}

// ---- search node ----------------------------------------------------------------
struct Node {
  int valid, x, y, w;
  int cy, cx, range, step, stages, count;
  int pr, pc, copy;
};

#define ME_COARSE_STEP 4
#define ME_REFINE 3

__device__ __forceinline__ int leaf_no8(const FrameParams *fp) {
  return (fp->turbo & T_LEAF_NO8) && fp->leaf && !fp->frame_is_intra;
}

// Node setup (k_me.h:141-178).
__device__ __forceinline__ Node make_node(const FrameParams *fp, int sb, int level, int i, const int32_t *mv) {
  Node m;
  int sbRow = sb / fp->sb_cols, sbCol = sb % fp->sb_cols, n = 1 << level;
  m.w = 64 >> level;
  const int iy = i >> level, ix = i & (n - 1);
  m.x = sbCol * 64 + ix * m.w;
  m.y = sbRow * 64 + iy * m.w;
  m.valid = m.x < fp->frame_w && m.y < fp->frame_h;
  m.cy = m.cx = 0;
  m.range = fp->me_range;
  m.pr = m.pc = 0;
  m.copy = 0;
  if (level > 0) {
    int pi = (iy >> 1) * (n >> 1) + (ix >> 1);
    const int32_t *par = mv + (sb * NUM_NODES + node_base(level - 1) + pi) * 2;
    m.pr = par[0];
    m.pc = par[1];
    m.cy = m.pr >> 3;
    m.cx = m.pc >> 3;
    m.range = imin(m.range, (fp->turbo & T_ME_CR1) ? 1 : (fp->turbo & T_ME_CR2) ? 2 : 4);
    m.copy = ((fp->turbo & T_ME_L3COPY) || leaf_no8(fp)) && level == 3;
  }
  m.step = 1;
  m.stages = 1;
  if (level == 0) {
    m.step = (fp->turbo & T_ME_HME3) ? 2 * ME_COARSE_STEP : ME_COARSE_STEP;
    m.range = (m.range / m.step) * m.step;
    m.stages = (fp->turbo & T_ME_HME3) ? 3 : 2;
  }
  if (level == 3 && (fp->turbo & T_ME_L3SUB)) m.stages = 0;
  int side = 2 * (m.range / m.step) + 1;
  m.count = 1 + side * side;
  return m;
}

// Later stages of level 0 (k_me.h:182-194).
__device__ void refine_stage(const FrameParams *fp, Node *m, int wy, int wx, int stage) {
  m->cy = wy;
  m->cx = wx;
  if (stage == 1 && (fp->turbo & T_ME_HME3)) {
    m->range = ME_COARSE_STEP;
    m->step = ME_COARSE_STEP;
  } else {
    m->range = (fp->turbo & T_ME_REF2) ? 2 : ME_REFINE;
    m->step = 1;
  }
  int side = 2 * (m->range / m->step) + 1;
  m->count = 1 + side * side;
}

// Candidate k of the current stage: 0 the centre, then the grid in raster order.
__device__ __forceinline__ void candidate(const Node &m, int k, int *dy, int *dx) {
  if (k == 0) {
    *dy = m.cy;
    *dx = m.cx;
    return;
  }
  k -= 1;
  int side = 2 * (m.range / m.step) + 1;
  *dy = m.cy - m.range + (k / side) * m.step;
  *dx = m.cx - m.range + (k % side) * m.step;
}

__device__ __forceinline__ uint32_t load_u32_unaligned(const uint8_t *p) {
  uintptr_t a = (uintptr_t)p;
  const uint32_t *q = (const uint32_t *)(a & ~(uintptr_t)3);
  uint32_t lo = __ldg(q), hi = __ldg(q + 1);
  return __funnelshift_r(lo, hi, (unsigned)(a & 3) * 8);
}

// Full-pel SAD of the w x w block at (x, y) against the reference at offset
// (dy, dx), rows strided by rs, scaled back by rs; reference coordinates
// clamped to the frame (k_me.h:39-64).
__device__ int full_sad(const Frame &f, const Node &m, int dy, int dx, int rs) {
  const FrameParams *fp = f.fp;
  int stride = fp->stride[0], W = fp->frame_w, Hh = fp->frame_h;
  const uint8_t *src = f.src + fp->offset[0], *ref = f.ref + fp->offset[0];
  int w = m.w, x = m.x, y = m.y;
  unsigned sad = 0;
  if (x + dx >= 0 && x + dx + w <= W && y + dy >= 0 && y + dy + w <= Hh) {
    for (int i = 0; i < w; i += rs) {
      const uint32_t *s = (const uint32_t *)(src + (y + i) * stride + x);
      const uint8_t *r = ref + (y + i + dy) * stride + x + dx;
      for (int j = 0; j < (w >> 2); j++) sad = __vsadu4(__ldg(s + j), load_u32_unaligned(r + 4 * j)) + sad;
    }
    return (int)sad * rs;
  }
  for (int i = 0; i < w; i += rs) {
    int ry = clip3(0, Hh - 1, y + i + dy);
    const uint8_t *s = src + (y + i) * stride + x;
    const uint8_t *r = ref + ry * stride;
    for (int j = 0; j < w; j++) sad += iabs((int)s[j] - (int)r[clip3(0, W - 1, x + j + dx)]);
  }
  return (int)sad * rs;
}

// SAD x16 on the decimated planes at offset (dy, dx), multiples of 4 (k_me.h:121-130).
__device__ int dec_sad(const Frame &f, const Node &m, int dy, int dx) {
  const FrameParams *fp = f.fp;
  int W = dec_w(fp), H = dec_h(fp), n = m.w >> 2, x0 = m.x >> 2, y0 = m.y >> 2, oy = dy >> 2, ox = dx >> 2, sad = 0;
  for (int i = 0; i < n; i++) {
    int sy = imin(y0 + i, H - 1), ry = clip3(0, H - 1, y0 + i + oy);
    for (int j = 0; j < n; j++)
      sad += iabs((int)f.dsrc[sy * W + imin(x0 + j, W - 1)] - (int)f.dref[ry * W + clip3(0, W - 1, x0 + j + ox)]);
  }
  return sad * 16;
}

// Rate of a full-pel vector (k_me.h:211-220).
__device__ __forceinline__ int mv_cost(const FrameParams *fp, int dy, int dx) {
  int bits = 2 + 2 * (31 - __clz(iabs(dy) * 8 + 1)) + 2 * (31 - __clz(iabs(dx) * 8 + 1));
  return fp->ac_q[0] * bits / 64;
}

// Full-pel cost (k_me.h:211-220).
__device__ __noinline__ int full_cost(const Frame f, const Node m, int dy, int dx) {
  const FrameParams *fp = f.fp;
  if ((fp->turbo & T_ME_DEC) && m.step >= ME_COARSE_STEP) return dec_sad(f, m, dy, dx) + mv_cost(fp, dy, dx);
  int rs = (fp->turbo & T_ME_RSUB) && m.step == 1 ? 2 : 1;
  return full_sad(f, m, dy, dx, rs) + mv_cost(fp, dy, dx);
}

// The same cost with the warp's 32 lanes splitting one candidate's byte pairs
// (levels of few nodes, a CTA each: its warps take candidates in
// turn instead of one thread a candidate). Every lane returns the total. The
// sums are the ones full_sad / dec_sad form, in another order: unsigned
// integer addition, so the cost is the same.
// Not inlined, with its arguments by value: the kernel's other parts keep
// their registers. The node width is a constant: as an argument it cost the
// whole search of a 3840x2160 picture 5,938 us against 4,994, of a 640x360 one
// 693 against 531 (full sums, +-64 samples).
template <int w>
__device__ __noinline__ int warp_full_cost(const FrameParams *fp, const uint8_t *fsrc, const uint8_t *fref,
                                           const uint8_t *dsrc, const uint8_t *dref, int x, int y, int step,
                                           int dy, int dx, int lane) {
  constexpr int lg = w == 64 ? 4 : w == 32 ? 3 : 2, n = 1 << lg;  // words of a row, and pairs of a decimated one
  unsigned sad = 0;
  int scale;
  if ((fp->turbo & T_ME_DEC) && step >= ME_COARSE_STEP) {
    // dec_sad: n x n pairs of the decimated planes, lanes along rows
    int W = dec_w(fp), H = dec_h(fp);
    int x0 = x >> 2, y0 = y >> 2, oy = dy >> 2, ox = dx >> 2;
    if (x0 + n + 4 <= W && y0 + n <= H && x0 + ox >= 0 && x0 + ox + n + 4 <= W && y0 + oy >= 0 && y0 + oy + n <= H) {
      // inside, with the words around a row's ends: four pairs a word
      for (int p = lane; p < n * n >> 2; p += 32) {
        int i = p >> (lg - 2), j = (p & ((n >> 2) - 1)) * 4;
        sad = __vsadu4(load_u32_unaligned(dsrc + (y0 + i) * W + x0 + j), load_u32_unaligned(dref + (y0 + i + oy) * W + x0 + ox + j)) + sad;
      }
    } else
    for (int p = lane; p < n * n; p += 32) {
      int i = p >> lg, j = p & (n - 1);
      int sy = imin(y0 + i, H - 1), ry = clip3(0, H - 1, y0 + i + oy);
      sad = __sad((int)dsrc[sy * W + imin(x0 + j, W - 1)], (int)dref[ry * W + clip3(0, W - 1, x0 + j + ox)], sad);
    }
    scale = 16;
  } else {
    // full_sad: rows 0, rs, 2 rs, ... of w / 4 words, lanes along rows
    int rs = (fp->turbo & T_ME_RSUB) && step == 1 ? 2 : 1;
    int stride = fp->stride[0], W = fp->frame_w, Hh = fp->frame_h;
    const uint8_t *src = fsrc + fp->offset[0], *ref = fref + fp->offset[0];
    const int nw = (w / rs) << lg;
    if (x + dx >= 0 && x + dx + w <= W && y + dy >= 0 && y + dy + w <= Hh) {
      for (int q = lane; q < nw; q += 32) {
        int i = (q >> lg) * rs, j = q & (n - 1);
        uint32_t s = __ldg((const uint32_t *)(src + (y + i) * stride + x) + j);
        sad = __vsadu4(s, load_u32_unaligned(ref + (y + i + dy) * stride + x + dx + 4 * j)) + sad;
      }
    } else {
      for (int q = lane; q < nw; q += 32) {
        int i = (q >> lg) * rs, j = q & (n - 1);
        const uint8_t *s = src + (y + i) * stride + x + 4 * j;
        const uint8_t *r = ref + clip3(0, Hh - 1, y + i + dy) * stride;
        for (int b = 0; b < 4; b++) sad = __sad((int)s[b], (int)r[clip3(0, W - 1, x + 4 * j + b + dx)], sad);
      }
    }
    scale = rs;
  }
  sad = __reduce_add_sync(0xffffffffu, sad);
  return (int)sad * scale + mv_cost(fp, dy, dx);
}

// The full-pel refinement of +-2 samples around (cy, cx) with every candidate
// inside the frame: `part` of `parts` warps takes its share of the node's
// words, one word position a lane at a time. A position's 25 candidates read
// 5 rows of 3 words (a candidate a lane read 2 unaligned words each, from
// scattered rows) and the 25 sums are reduced over the warp; lane k returns
// candidate k's part (0: the centre, 1 + raster index: the grid).
__device__ __forceinline__ bool grid_inside(const FrameParams *fp, const Node &m) {
  return m.step == 1 && m.range == 2 && m.x + m.cx >= 2 && m.y + m.cy >= 2 && m.x + m.cx + 2 + m.w <= fp->frame_w &&
         m.y + m.cy + 2 + m.w <= fp->frame_h;
}
template <int w, int parts>
__device__ __noinline__ unsigned grid_sads(const FrameParams *fp, const uint8_t *fsrc, const uint8_t *fref, int x, int y, int cy,
                                           int cx, int rs, int lane, int part) {
  constexpr int lgw = w == 64 ? 4 : w == 32 ? 3 : 2;
  const int stride = fp->stride[0], n = (w / rs) << lgw;
  const uint8_t *src = fsrc + fp->offset[0] + y * stride + x;
  const uint8_t *ref = fref + fp->offset[0] + (y + cy - 2) * stride + x + cx - 2;
  const int off = (int)((uintptr_t)ref & 3);
  ref -= off;
  unsigned sad[25];
#pragma unroll
  for (int k = 0; k < 25; k++) sad[k] = 0;
  for (int q = lane + part * 32; q < n; q += 32 * parts) {
    const int i = (q >> lgw) * rs, j = (q & ((1 << lgw) - 1)) * 4;
    const uint32_t sv = __ldg((const uint32_t *)(src + i * stride + j));
#pragma unroll
    for (int dy = 0; dy < 5; dy++) {
      const uint32_t *p = (const uint32_t *)(ref + (i + dy) * stride + j);
      const uint32_t a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
      // bytes -2 .. 5 around the word
      const uint32_t lo = __funnelshift_r(a, b, 8 * off), hi = __funnelshift_r(b, c, 8 * off);
      sad[dy * 5] = __vsadu4(sv, lo) + sad[dy * 5];
#pragma unroll
      for (int dx = 1; dx < 4; dx++) sad[dy * 5 + dx] = __vsadu4(sv, __funnelshift_r(lo, hi, 8 * dx)) + sad[dy * 5 + dx];
      sad[dy * 5 + 4] = __vsadu4(sv, hi) + sad[dy * 5 + 4];
    }
  }
  unsigned mine = 0;
#pragma unroll
  for (int k = 0; k < 25; k++) {
    unsigned v = __reduce_add_sync(0xffffffffu, sad[k]);
    if (lane == 1 + k || (k == 12 && lane == 0)) mine = v;
  }
  return mine * rs;
}

// A row's 4-point Hadamard transform is four dot products of its bytes with
// +-1 words; `h` picks the word.
__host__ __device__ constexpr uint32_t hadamard_word(int h) {
  return h == 0 ? 0x01010101u : h == 1 ? 0xffff0101u : h == 2 ? 0x01ffff01u : 0xff01ff01u;  // ++++, ++--, +--+, +-+-
}
__host__ __device__ constexpr uint32_t hadamard_minus(int h) {
  return h == 0 ? 0xffffffffu : h == 1 ? 0x0101ffffu : h == 2 ? 0xff0101ffu : 0x01ff01ffu;
}

// SATD of the 4x4 unit at (ux, uy) against the quarter-pel plane prediction at
// (mvr, mvc) (even, 1/8 units) (k_me.h:317-340). S: the source rows'
// transforms, formed once for all of a unit's candidates; a candidate's rows
// are then 16 dot products, without unpacking a sample.
__device__ __forceinline__ int unit_satd_hp(const uint8_t *qp, size_t planeSize, int W, int H, int ux, int uy, const int (&S)[16],
                                            int mvr, int mvc) {
  const uint8_t *pl = qp + (size_t)(((mvr >> 1) & 3) * 4 + ((mvc >> 1) & 3)) * planeSize;
  const int iy = uy + (mvr >> 3), ix = ux + (mvc >> 3);
  uint32_t pv[4];
  if (ix >= 0 && ix + 8 <= W && iy >= 0 && iy + 4 <= H) {
    // inside the plane, and the two aligned words each row load stay in the row: no clamping
    const uint8_t *a = pl + (size_t)iy * W + ix;
    if ((W & 3) == 0) {
      const int off = (int)((uintptr_t)a & 3);
      const uint32_t *q = (const uint32_t *)(a - off);
#pragma unroll
      for (int r = 0; r < 4; r++) pv[r] = __funnelshift_r(__ldg(q + r * (W >> 2)), __ldg(q + r * (W >> 2) + 1), 8 * off);
    } else {
#pragma unroll
      for (int r = 0; r < 4; r++) pv[r] = load_u32_unaligned(a + (size_t)r * W);
    }
  } else {
    for (int r = 0; r < 4; r++) {
      const uint8_t *row = pl + (size_t)clip3(0, H - 1, iy + r) * W;
      uint32_t v = 0;
      for (int c = 0; c < 4; c++) v |= (uint32_t)row[clip3(0, W - 1, ix + c)] << (8 * c);
      pv[r] = v;
    }
  }
  int sum = 0;
#pragma unroll
  for (int h = 0; h < 4; h++) {
    int t[4];
#pragma unroll
    for (int r = 0; r < 4; r++) t[r] = dp4s(pv[r], hadamard_minus(h), S[4 * h + r]);
    // |a + c| + |a - c| = 2 max(|a|, |c|)
    sum += imax(iabs(t[0] + t[1]), iabs(t[2] + t[3])) + imax(iabs(t[0] - t[1]), iabs(t[2] - t[3]));
  }
  return 2 * sum;
}

// SATD of 4x4 unit u against the normative EIGHTTAP prediction of the node
// at (mvr, mvc) (the non-plane path, k_me.h:254-257).
__device__ __noinline__ int unit_satd_pred(const Frame f, const Node m, int mvr, int mvc, int u) {
  const FrameParams *fp = f.fp;
  const int ln = 31 - __clz(m.w >> 2), bx = (u & ((1 << ln) - 1)) * 4, by = (u >> ln) * 4;
  pred::Inter p;
  pred::inter_setup(&p, f.ref + fp->offset[0], fp->stride[0], fp->frame_w, fp->frame_h, m.x, m.y, m.w, m.w, mvr, mvc,
                    0, 0, EIGHTTAP);
  const uint8_t *sp = f.src + fp->offset[0] + (m.y + by) * fp->stride[0] + m.x + bx;
  int d[16];
  pred::inter_unit4(&p, by, bx, d);
  for (int r = 0; r < 4; r++) {
    uint32_t sv = __ldg((const uint32_t *)(sp + r * fp->stride[0]));  // units start on words
    for (int c = 0; c < 4; c++) d[r * 4 + c] = (int)((sv >> (8 * c)) & 255) - d[r * 4 + c];
  }
  return pred::satd4x4(d);
}

__device__ __forceinline__ void sub_neighbour(const FrameParams *fp, int j, int step, int *dr, int *dc) {
  int k = (fp->turbo & T_ME_CROSS) ? (j == 0 ? 1 : j == 1 ? 3 : j == 2 ? 4 : 6) : j;
  *dr = (k < 3) ? -step : (k < 5 ? 0 : step);
  *dc = (k == 0 || k == 3 || k == 5) ? -step : ((k == 1 || k == 6) ? 0 : step);
}

// The threads searching one node (me_group): a CTA, a warp, or half a warp (the
// 8x8 level, whose nodes have at most 16 sub-pel pairs at a time); mask holds
// the group's lanes of its warp.
template <int SIZE>
struct MeGrp {
  static constexpr int size = SIZE;
  int rank;
  unsigned mask;
  __device__ __forceinline__ void sync() const {
    if (size > 32) __syncthreads();
    else __syncwarp(mask);
  }
};

// Minimum over the group's lanes of its warp (the whole warp for a CTA group).
template <class Grp>
__device__ __forceinline__ unsigned long long group_min(unsigned long long v, const Grp &g) {
  for (int off = g.size >= 32 ? 16 : g.size >> 1; off > 0; off >>= 1) {
    unsigned long long o = __shfl_xor_sync(g.mask, v, off);
    v = o < v ? o : v;
  }
  return v;
}

// Sub-pel costs of ncand candidates (mvr[c], mvc[c]) into cost[c] (shared,
// private to the group), every (candidate, unit) pair spread over the group.
// ST: every ST-th unit counts.
template <int LEVEL, bool HP, int ST, class Grp>
__device__ __forceinline__ void subpel_costs(const Frame &f, const Node &m, const int *cr, const int *cc, int ncand, int *cost,
                                             const Grp &g) {
  const FrameParams *fp = f.fp;
  constexpr int st = ST, ln = 4 - LEVEL, nus = (1 << (2 * ln)) / ST;
  if (g.rank == 0) WORK(W_ME_SATD, ncand * nus);
  const int W = fp->frame_w, H = fp->frame_h, ss = fp->stride[0];
  const size_t planeSize = (size_t)W * H;
  // unit u of the node (every st-th counts): its place and, with planes, its source rows' transforms
  int ux = 0, uy = 0;
  int S[16];
  auto take = [&](int u) {
    ux = m.x + ((u * st) & ((1 << ln) - 1)) * 4;
    uy = m.y + ((u * st) >> ln) * 4;
    if (HP)
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const uint32_t v = __ldg((const uint32_t *)(f.src + fp->offset[0] + (uy + r) * ss + ux));
#pragma unroll
        for (int h = 0; h < 4; h++) S[4 * h + r] = dp4s(v, hadamard_word(h), 0);
      }
  };
  auto satd = [&](int c, int u) {
    return HP ? unit_satd_hp(f.qp, planeSize, W, H, ux, uy, S, cr[c], cc[c]) : unit_satd_pred(f, m, cr[c], cc[c], u * st);
  };
  if constexpr (nus >= Grp::size) {
    // a candidate at a time, its units over the group (both powers of two)
    if (g.size > 32) {
      if (g.rank < ncand) cost[g.rank] = 0;
      g.sync();
    }
    constexpr bool one = nus == Grp::size;  // a unit a thread, the same for every candidate
    if (one) take(g.rank);
    for (int c = 0; c < ncand; c++) {
      int v = 0;
      for (int u = g.rank; u < nus; u += g.size) {
        if (!one) take(u);
        v += satd(c, u);
      }
      v = __reduce_add_sync(g.mask, v);
      if (g.size > 32) {
        if ((g.rank & 31) == 0) atomicAdd(&cost[c], v * st);
      } else if (g.rank == 0) {
        cost[c] = v * st;
      }
    }
  } else if constexpr (nus >= 32) {
    // several candidates at a time, nus / 32 warps of the CTA each
    if (g.rank < ncand) cost[g.rank] = 0;
    g.sync();
    const int u = g.rank & (nus - 1);
    take(u);
    for (int c = g.rank / nus; c < ncand; c += Grp::size / nus) {
      int v = __reduce_add_sync(g.mask, satd(c, u));
      if ((g.rank & 31) == 0) atomicAdd(&cost[c], v * st);
    }
  } else {
    // several candidates at a time, nus lanes each
    constexpr int lg = 2 * ln;
    const int u = g.rank & (nus - 1);
    take(u);
    for (int c = g.rank >> lg; c < ((ncand << lg) + g.size - 1) / g.size * (g.size >> lg); c += g.size >> lg) {
      int v = c < ncand ? satd(c, u) : 0;
      for (int o = nus >> 1; o; o >>= 1) v += __shfl_xor_sync(g.mask, v, o);
      if (c < ncand && u == 0) cost[c] = v * st;
    }
  }
  g.sync();
}

// One search level: a whole CTA per node (few, large nodes), a warp per (node,
// reference), or half a warp (the 8x8 level);
// blockIdx.y selects the reference. Level and sub-pel path (HP: quarter-pel
// planes) are compile-time: with one kernel for all of them the 16x16 level
// executed 3,800 instructions a node, a seventh of them spilled registers.
// 6 CTAs per SM with planes (80 registers a thread; 1-2% on the 1080p clip over
// 5), 5 without (96 registers, of which the prediction spills up to 208 bytes a
// thread at the 8x8 level).
// Without planes every full-range candidate is a full SAD and every sub-pel
// unit its own prediction, and a picture has few large nodes (640x360: 60 and
// 240): 16 warps take a 64x64 node and 4 a 32x32 one.
// The whole search of a frame, 4 warps and 1 against this, +-64 samples and +-32:
// 640x360 920 -> 531 us and 573 -> 338, 1920x1080 1,815 -> 1,543 and 1,125 -> 961,
// 3840x2160, where the nodes nearly fill the chip anyway, 5,190 -> 4,994 and
// 3,121 -> 3,078.
__host__ __device__ constexpr int me_group(int level, bool hp) {
  return level == 0 ? (hp ? 128 : 512) : level == 1 && !hp ? 128 : level == 3 ? 16 : 32;
}
__host__ __device__ constexpr int me_threads(int level, bool hp) { return level == 0 && !hp ? 512 : 128; }
template <int LEVEL, bool HP>
__global__ void __launch_bounds__(me_threads(LEVEL, HP), HP ? 6 : LEVEL == 0 ? 1 : 5) k_me_level(Frame f0, Frame f1) {
  __shared__ int s_cost[8][16];
  __shared__ int s_r[8][16], s_c[8][16];
  constexpr int group = me_group(LEVEL, HP), warps = me_threads(LEVEL, HP) / 32;
  constexpr bool whole_cta = group == 32 * warps;
  __shared__ unsigned long long s_best[warps];
  __shared__ unsigned s_sad[warps][26];
  const Frame f = blockIdx.y ? f1 : f0;
  const FrameParams *fp = f.fp;
  constexpr int level = LEVEL;
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = lane >> 4;
  const MeGrp<group> grp = whole_cta ? MeGrp<group>{(int)threadIdx.x, 0xffffffffu}
                           : group == 32 ? MeGrp<group>{lane, 0xffffffffu}
                                         : MeGrp<group>{lane & 15, 0xffffu << (16 * half)};
  int slotw = whole_cta ? 0 : group == 32 ? warp : 2 * warp + half;
  int nn = 1 << (2 * level);
  int g = whole_cta ? (int)blockIdx.x : (int)blockIdx.x * (128 / group) + slotw;
  if (g >= fp->sb_cols * fp->sb_rows * nn) return;
  int sb = g >> (2 * level), i = g & (nn - 1);
  Node m = make_node(fp, sb, level, i, f.mv);
  if (f.isGold && level == 3 && (fp->turbo & T_ME_G3COPY) && fp->leaf && !fp->frame_is_intra) m.copy = 1;
  int32_t *out = f.mv + (sb * NUM_NODES + node_base(level) + i) * 2;
  if (!m.valid) {
    if (grp.rank == 0) out[0] = out[1] = 0;
    return;
  }
  if (m.copy) {
    if (grp.rank == 0) {
      out[0] = m.pr;
      out[1] = m.pc;
    }
    return;
  }
  int by = 0, bx = 0;
  for (int stage = 0; stage < m.stages; stage++) {
    if (stage > 0) refine_stage(fp, &m, by, bx, stage);
    if (grp.rank == 0) {  // byte pairs of the stage's candidates (full_cost)
      int dec = (fp->turbo & T_ME_DEC) && m.step >= ME_COARSE_STEP, rs = (fp->turbo & T_ME_RSUB) && m.step == 1 ? 2 : 1;
      WORK(dec ? W_ME_DSAD : W_ME_SAD, (long long)m.count * (dec ? (m.w >> 2) * (m.w >> 2) : (m.w / rs) * m.w));
    }
    unsigned long long best = ~0ull;
    const int grs = (fp->turbo & T_ME_RSUB) ? 2 : 1;
    if (grp.size >= 32 && grid_inside(fp, m)) {
      unsigned sad = grid_sads<(64 >> LEVEL), whole_cta ? warps : 1>(fp, f.src, f.ref, m.x, m.y, m.cy, m.cx, grs, lane, whole_cta ? warp : 0);
      if (whole_cta) {
        if (lane < 26) s_sad[warp][lane] = sad;
        __syncthreads();
        sad = 0;
        if (lane < 26)
          for (int w = 0; w < warps; w++) sad += s_sad[w][lane];
      }
      if (lane < 26) {
        int dy, dx;
        candidate(m, lane, &dy, &dx);
        best = ((unsigned long long)((int)sad + mv_cost(fp, dy, dx)) << 32) | (unsigned)lane;
      }
    } else if (whole_cta) {
      // a warp per candidate, every lane holding the warp's running minimum
      for (int k = warp; k < m.count; k += warps) {
        int dy, dx;
        candidate(m, k, &dy, &dx);
        int cost = warp_full_cost<(64 >> LEVEL)>(fp, f.src, f.ref, f.dsrc, f.dref, m.x, m.y, m.step, dy, dx, lane);
        unsigned long long key = ((unsigned long long)(unsigned)cost << 32) | (unsigned)k;
        best = key < best ? key : best;
      }
    } else {
      for (int k = grp.rank; k < m.count; k += grp.size) {
        int dy, dx;
        candidate(m, k, &dy, &dx);
        int cost;
        if (LEVEL == 3 && grs == 2 && m.x + dx >= 0 && m.x + dx + 8 <= fp->frame_w && m.y + dy >= 0 && m.y + dy + 8 <= fp->frame_h) {
          // full_sad of every second row of an 8x8 node inside the frame
          const int stride = fp->stride[0];
          const uint8_t *sp = f.src + fp->offset[0] + m.y * stride + m.x, *rp = f.ref + fp->offset[0] + (m.y + dy) * stride + m.x + dx;
          const int off = (int)((uintptr_t)rp & 3);
          rp -= off;
          unsigned sad = 0;
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            const uint32_t *sw = (const uint32_t *)(sp + i * stride), *rw = (const uint32_t *)(rp + i * stride);
            const uint32_t a = __ldg(rw), b = __ldg(rw + 1), c = __ldg(rw + 2);
            sad = __vsadu4(__ldg(sw), __funnelshift_r(a, b, 8 * off)) + sad;
            sad = __vsadu4(__ldg(sw + 1), __funnelshift_r(b, c, 8 * off)) + sad;
          }
          cost = (int)sad * 2 + mv_cost(fp, dy, dx);
        } else {
          cost = full_cost(f, m, dy, dx);
        }
        unsigned long long key = ((unsigned long long)(unsigned)cost << 32) | (unsigned)k;
        best = key < best ? key : best;
      }
    }
    best = group_min(best, grp);
    if (whole_cta) {
      __syncthreads();
      if (lane == 0) s_best[warp] = best;
      __syncthreads();
      for (int w = 0; w < warps; w++) best = s_best[w] < best ? s_best[w] : best;
    }
    candidate(m, (int)(best & 0xffffffffu), &by, &bx);
  }
  if (level > 0 && (m.copy || ((fp->turbo & T_ME_KEEP) && by == m.cy && bx == m.cx))) {
    if (grp.rank == 0) {
      out[0] = m.pr;
      out[1] = m.pc;
    }
    return;
  }
  // sub-pel refinement (k_me.h:262-281)
  int *cost = s_cost[slotw], *cr = s_r[slotw], *cc = s_c[slotw];
  int mvr = m.stages ? by * 8 : m.pr, mvc = m.stages ? bx * 8 : m.pc;
  if (grp.rank == 0) {
    cr[0] = mvr;
    cc[0] = mvc;
  }
  grp.sync();
  auto costs = [&](int ncand) {
    // large nodes may count every second unit
    if (HP && LEVEL < 2 && (fp->turbo & T_ME_USUB)) subpel_costs<LEVEL, HP, LEVEL < 2 ? 2 : 1>(f, m, cr, cc, ncand, cost, grp);
    else subpel_costs<LEVEL, HP, 1>(f, m, cr, cc, ncand, cost, grp);
  };
  costs(1);
  int bestS = cost[0];
  int minStep = m.w >= 32 && (fp->turbo & T_ME_HALF01) ? 4 : 2;
  int nb = (fp->turbo & T_ME_CROSS) ? 4 : 8;
  for (int step = 4; step >= minStep; step >>= 1) {
    grp.sync();
    if (grp.rank < nb) {
      int dr, dc;
      sub_neighbour(fp, grp.rank, step, &dr, &dc);
      cr[grp.rank] = mvr + dr;
      cc[grp.rank] = mvc + dc;
    }
    grp.sync();
    costs(nb);
    // running strict minimum over the neighbours in order == first minimum
    int bk = -1, bc = bestS;
    for (int k = 0; k < nb; k++)
      if (cost[k] < bc) {
        bc = cost[k];
        bk = k;
      }
    if (bk >= 0) {
      bestS = bc;
      mvr = cr[bk];
      mvc = cc[bk];
    }
  }
  if (grp.rank == 0) {
    out[0] = mvr;
    out[1] = mvc;
  }
}

}  // namespace me
