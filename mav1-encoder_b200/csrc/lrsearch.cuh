// Loop-restoration parameter search on the device: the reference's lr_select
// (src/lr_search.c:244-359) with its Wiener least-squares fit (wiener_fit,
// :142-193), its self-guided projection fit (sgr_fit, :196-240), the unit SSE
// (unit_sse, :92-108) and the rate of the unit parameters (lr_unit_params /
// lr_subexp, :33-80).
//
// Per restoration unit the reference compares RESTORE_NONE, a fitted Wiener
// filter refined greedily by +-1 tap steps, and every self-guided set with
// fitted projection weights, by 16 * SSE + lambda * bits. The rate of a unit's
// parameters depends on the parameters the previous unit of the plane chose
// (subexponential coding against running references), so the choice is a
// serial scan over the units. Everything that does not depend on those
// references is computed first, for all units at once:
//
//   k_lr_fit     three CTAs per unit: the SSE of RESTORE_NONE, the Wiener fit,
//                the SSE of the fitted filter and of its single-tap
//                neighbours (the candidates the refinement tries first); and
//                for half of the self-guided sets each the fit and its SSE;
//   k_lr_spec    one CTA per unit: the Wiener refinement replayed under
//                guessed running references, caching the SSE of every
//                candidate it visits (SSEs do not depend on the references);
//   k_lr_choose  a warp per unit: lr_select's rate comparisons under guessed
//                running references, twice;
//   k_lr_select  one CTA per plane: the units whose references turned out
//                different are chosen again, until every unit stands; a
//                refinement candidate whose SSE no pass cached is evaluated on
//                the spot by the whole CTA, for units with settled references.
//
// Bit-exactness. SSEs, the self-guided sums and the first Wiener iteration
// are integer-valued (every partial sum is an integer below 2^53, so double
// and int64 sums agree in any order). The later Wiener iterations accumulate
// non-integer doubles: they are summed in the reference's order (the unit's
// 4x4 blocks in raster order, each block's samples in raster order) by one
// lane per accumulator, and every double operation is the reference's, in
// its order, with explicit round-to-nearest intrinsics (no contraction into
// fused multiply-adds). lround is restated as round-half-away-from-zero.
#pragma once

#include "common.cuh"
#include "filters.cuh"

namespace lrs {

constexpr int THREADS = 256;
constexpr int CACHE = 40;       // candidate SSEs a unit keeps from the first pass and the speculative pass
constexpr int MIN_CACHE = 25;   // the first pass's 13 at most, and the 12 a path under settled references can add
constexpr int LIST = 256;       // units k_lr_select chooses again in a round

// What the first pass leaves for the serial choice, per unit.
struct Fit {
  long long sse_none;
  int w[2][3];                  // fitted Wiener taps
  int n, n0;                    // cached Wiener candidates; those of the first pass
  int taps[CACHE][6];           // their taps: pass 0 j 0..2, pass 1 j 0..2
  long long sse[CACHE];
  int xqd[16][2];               // fitted projection weights per self-guided set
  long long sgr_sse[16];
  int used[8];                  // the choice: running references it was made with (taps, projection weights)
};

// The unit's 4x4 luma block range: rows [r0, r1), columns [c0, c1) of the
// frame's 4x4 grid whose blocks lr_block_setup assigns to unit (ur, uc) of
// the plane (the counting sort of lr_select, lr_search.c:250-272, keeps them
// in raster order).
struct Geom {
  int plane, ur, uc, r0, r1, c0, c1;
};

HD int unit_row_of(const FrameParams *fp, int plane, int r) {
  return imin(fp->lr_unit_rows[plane] - 1, ((r * MI_SIZE + 8) >> (plane > 0)) / fp->lr_unit_size[plane]);
}
HD int unit_col_of(const FrameParams *fp, int plane, int c) {
  return imin(fp->lr_unit_cols[plane] - 1, ((c * MI_SIZE) >> (plane > 0)) / fp->lr_unit_size[plane]);
}

// First r in [0, n) with of(r) >= v, or n: unit_row_of / unit_col_of are
// non-decreasing in r (a clamped quotient of a growing numerator).
template <typename F>
__device__ __forceinline__ int first_at_least(int n, int v, F of) {
  int lo = 0, hi = n;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (of(mid) >= v) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

// The 4x4 rows and columns whose unit is (ur, uc): the contiguous run of r
// with unit_row_of(r) == ur (and the same for columns), found by binary
// search since the maps are non-decreasing; an empty run leaves
// r0 = rows4, r1 = 0 (c0 = cols4, c1 = 0).
__device__ void unit_geom(const FrameParams *fp, int plane, int ur, int uc, Geom *g) {
  int rows4 = (fp->frame_h + 3) >> 2, cols4 = (fp->frame_w + 3) >> 2;
  g->plane = plane;
  g->ur = ur;
  g->uc = uc;
  auto rowOf = [&](int r) { return unit_row_of(fp, plane, r); };
  auto colOf = [&](int c) { return unit_col_of(fp, plane, c); };
  int r0 = first_at_least(rows4, ur, rowOf), r1 = first_at_least(rows4, ur + 1, rowOf);
  int c0 = first_at_least(cols4, uc, colOf), c1 = first_at_least(cols4, uc + 1, colOf);
  g->r0 = r0 < r1 ? r0 : rows4;
  g->r1 = r0 < r1 ? r1 : 0;
  g->c0 = c0 < c1 ? c0 : cols4;
  g->c1 = c0 < c1 ? c1 : 0;
}

// A unit's samples in shared memory. A unit is cut into the stripes its rows
// fall in (a luma unit is one stripe, the last row of units up to two; a
// chroma unit two, up to four): `tap` holds, per stripe, the samples
// get_source_sample( ) returns over the stripe's rows and columns plus 3 on
// every side, with the clamps to the plane and the stripe's CDEF / deblocked
// choice already made, so the filters read it with plain indices. `src` holds
// the unit's source samples. Every other array of a pass is laid out behind
// them; Dims are the largest unit of the frame, so shared memory is no larger
// than the frame's units need (64 x 64 units: 93 KB, two CTAs per SM; the
// largest unit, 95 x 103, takes 222 KB).
constexpr int MAX_SEGS = 4, MAX_UNIT_W = 95, MAX_UNIT_H = 103;
struct Dims {
  int w, h;                 // largest width and height
  int rows6, rows2, odd;    // largest h + 6 segs, h + 2 segs, h / 2 + 2 segs
};
// units of 64 samples: a luma unit of up to 103 rows has two stripes, a chroma
// unit of up to 99 rows four
constexpr Dims MAX_DIMS = {MAX_UNIT_W, MAX_UNIT_H, 99 + 6 * 4, 103 + 2 * 2, 99 / 2 + 2 * 4};
HD int align16(int x) { return (x + 15) & ~15; }
struct Layout {
  int tap_p, src_p;                         // row pitches
  int tap, src;                             // byte offsets
  int p1, b1, p2, b2, ab1, ab2, fd, sgr_end;  // self-guided pass
  int hv, phi, wiener_end;                  // Wiener fit
};
HD Layout layout_of(const Dims &d) {
  Layout l;
  l.tap_p = (d.w + 6 + 3) & ~3;
  l.src_p = (d.w + 3) & ~3;
  l.tap = 0;
  l.src = align16(d.rows6 * l.tap_p);
  int base = align16(l.src + d.h * l.src_p);
  int n1 = d.rows2 * (d.w + 2), n2 = d.odd * (d.w + 2);
  l.p1 = base;
  l.b1 = align16(l.p1 + 4 * n1);
  l.p2 = align16(l.b1 + 2 * n1);
  l.b2 = align16(l.p2 + 4 * n2);
  l.ab1 = align16(l.b2 + 2 * n2);
  l.ab2 = align16(l.ab1 + 4 * n1);
  l.fd = align16(l.ab2 + 4 * n2);
  l.sgr_end = align16(l.fd + 4 * d.h * d.w);
  int nv = d.rows6 * d.w, nh = d.h * (d.w + 6);
  l.hv = base;
  l.phi = align16(l.hv + 8 * (nv > nh ? nv : nh));
  l.wiener_end = l.phi + 2 * 4 * d.w * 4 * 8;
  return l;
}
HD int smem_fit(const Layout &l) { return l.sgr_end > l.wiener_end ? l.sgr_end : l.wiener_end; }
HD int smem_sse(const Layout &l) { return l.p1; }

// The largest unit of the planes of a frame (the last unit of a row or column
// takes the remainder; unit rows start 8 luma rows early).
inline Dims unit_dims(const FrameParams &fp) {
  Dims d = {1, 1, 1, 1, 1};
  for (int p = 0; p < 3; p++) {
    int sub = p > 0, size = fp.lr_unit_size[p], off = 8 >> sub, stripe = 64 >> sub;
    int pw = (fp.frame_w + sub) >> sub, ph = (fp.frame_h + sub) >> sub;
    int rows = fp.lr_unit_rows[p], cols = fp.lr_unit_cols[p];
    d.w = imax(d.w, cols <= 1 ? pw : imax(size, pw - size * (cols - 1)));
    // the first row of units starts mid-stripe, later ones on a stripe when the size is a multiple of it
    int hs[2] = {rows <= 1 ? ph : size - off, rows <= 1 ? 0 : imax(size, ph - size * (rows - 1) + off)};
    for (int k = 0; k < 2; k++) {
      int h = hs[k], slack = k == 0 ? off : size % stripe ? stripe - 1 : 0;
      int segs = (h + slack + stripe - 1) / stripe;
      d.h = imax(d.h, h);
      d.rows6 = imax(d.rows6, h + 6 * segs);
      d.rows2 = imax(d.rows2, h + 2 * segs);
      d.odd = imax(d.odd, h / 2 + 2 * segs);
    }
  }
  return d;
}

// The unit a CTA works on: its plane samples x0 .. x0 + w - 1, rows y0 .. y0 +
// h - 1, cut into stripes: segment s covers rows y0 + seg[s] .. y0 + seg[s + 1]
// - 1. Row i of the unit (segment s) is row i + 6 s + 3 of `tap`.
struct Area {
  int plane, x0, y0, w, h, nseg, seg[MAX_SEGS + 1];
  unsigned inv_w, inv_w2, inv_w6;  // 2^24 / d rounded up, d = w, w + 2, w + 6 (quotient())
};
// k / d for d's rounded-up reciprocal inv = ceil(2^24 / d): exact while k < 2^24 / d (here k < 14,000 and d < 104; the
// product stays below 2^32, k / d being at most 127).
__device__ __forceinline__ int quotient(int k, unsigned inv) { return (int)((unsigned)k * inv >> 24); }

__device__ __forceinline__ int seg_of(const Area &a, int row) {
  int s = 0;
  while (s + 1 < a.nseg && row >= a.seg[s + 1]) s++;
  return s;
}

// Finds the unit's area (one thread).
__device__ void unit_area(const FrameParams *fp, const Geom &g, Area *a) {
  const int sub = g.plane > 0, bw = MI_SIZE >> sub, stripe = 64 >> sub, off = 8 >> sub;
  const int endX = ((fp->frame_w + sub) >> sub) - 1, endY = ((fp->frame_h + sub) >> sub) - 1;
  a->plane = g.plane;
  a->x0 = (g.c0 * MI_SIZE) >> sub;
  a->y0 = (g.r0 * MI_SIZE) >> sub;
  a->w = g.c1 > g.c0 ? imax(0, imin(endX, ((g.c1 - 1) * MI_SIZE >> sub) + bw - 1) - a->x0 + 1) : 0;
  a->h = g.r1 > g.r0 && a->w > 0 ? imax(0, imin(endY, ((g.r1 - 1) * MI_SIZE >> sub) + bw - 1) - a->y0 + 1) : 0;
  a->nseg = 0;
  for (int row = 0; row < a->h && a->nseg < MAX_SEGS;) {
    a->seg[a->nseg++] = row;
    row += stripe - (a->y0 + row + off) % stripe;
  }
  a->seg[a->nseg] = a->h;
  a->inv_w = ((1u << 24) + imax(a->w, 1) - 1) / imax(a->w, 1);
  a->inv_w2 = ((1u << 24) + a->w + 1) / (a->w + 2);
  a->inv_w6 = ((1u << 24) + a->w + 5) / (a->w + 6);
}

// Fills `tap` and `src` (the whole CTA).
__device__ void stage_unit(const FrameParams *fp, const Area &a, const uint8_t *cdef, const uint8_t *dbk,
                           const uint8_t *src, const Layout &l, uint8_t *smem) {
  const int p = a.plane, sub = p > 0, stride = fp->stride[p], off = fp->offset[p];
  const int endX = ((fp->frame_w + sub) >> sub) - 1, endY = ((fp->frame_h + sub) >> sub) - 1;
  const int nrow = a.h ? a.h + 6 * a.nseg : 0, W6 = a.w + 6;
  for (int k = threadIdx.x; k < nrow * W6; k += THREADS) {
    int tr = quotient(k, a.inv_w6), c = k - tr * W6, s = 0;
    while (s + 1 < a.nseg && tr >= a.seg[s + 1] + 6 * (s + 1)) s++;
    int row = a.y0 + tr - 6 * s - 3;                                  // plane row asked for
    int st = ((a.y0 + a.seg[s] + (8 >> sub)) / (64 >> sub)) * (64 >> sub) - (8 >> sub), en = st + (64 >> sub) - 1;
    int x = imax(0, imin(endX, a.x0 + c - 3)), y = imax(0, imin(endY, row));
    const uint8_t *b = cdef;
    if (y < st) {
      y = imax(st - 2, y);
      b = dbk;
    } else if (y > en) {
      y = imin(en + 2, y);
      b = dbk;
    }
    smem[l.tap + tr * l.tap_p + c] = b[off + y * stride + x];
  }
  for (int k = threadIdx.x; k < a.h * a.w; k += THREADS) {
    int r = quotient(k, a.inv_w), c = k - r * a.w;
    smem[l.src + r * l.src_p + c] = src[off + (a.y0 + r) * stride + a.x0 + c];
  }
  __syncthreads();
}

// ---- double arithmetic exactly as the reference's C (no contraction) ---------
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }
// C lround: the nearest integer, halfway cases away from zero.
__device__ __forceinline__ long long lround_away(double x) {
  double t = trunc(x);
  if (fabs(dsub(x, t)) >= 0.5) t = dadd(t, x < 0 ? -1.0 : 1.0);
  return (long long)t;
}

// Gaussian elimination with partial pivoting (solve, lr_search.c:111-138).
__device__ int solve(int n, double M[3][3], double v[3], double *x) {
  for (int i = 0; i < n; i++) {
    int p = i;
    for (int r = i + 1; r < n; r++)
      if (fabs(M[r][i]) > fabs(M[p][i])) p = r;
    if (fabs(M[p][i]) < 1e-9) return 0;
    if (p != i) {
      for (int k = 0; k < n; k++) {
        double t = M[i][k];
        M[i][k] = M[p][k];
        M[p][k] = t;
      }
      double t = v[i];
      v[i] = v[p];
      v[p] = t;
    }
    for (int r = i + 1; r < n; r++) {
      double f = ddiv(M[r][i], M[i][i]);
      for (int k = i; k < n; k++) M[r][k] = dsub(M[r][k], dmul(f, M[i][k]));
      v[r] = dsub(v[r], dmul(f, v[i]));
    }
  }
  for (int i = n - 1; i >= 0; i--) {
    double s = v[i];
    for (int k = i + 1; k < n; k++) s = dsub(s, dmul(M[i][k], x[k]));
    x[i] = ddiv(s, M[i][i]);
  }
  return 1;
}

// ---- rate of the unit parameters (lr_subexp / lr_unit_params) -------------------
HD int recenter_nonneg(int r, int v) {
  if (v > (r << 1)) return v;
  if (v >= r) return (v - r) << 1;
  return ((r - v) << 1) - 1;
}

// bits of v coded as decode_signed_subexp_with_ref_bool( low, high, k, r )
HD int subexp_bits(int low, int high, int k, int r, int v) {
  int mx = high - low;
  r -= low;
  v -= low;
  int x = (r << 1) <= mx ? recenter_nonneg(r, v) : recenter_nonneg(mx - 1 - r, mx - 1 - v);
  int bits = 0, i = 0, mk = 0;
  for (;;) {
    int b2 = i ? k + i - 1 : k;
    int a = 1 << b2;
    if (mx <= mk + 3 * a) {
      int n = mx - mk, val = x - mk;
      int w = floor_log2(n) + 1, m = (1 << w) - n;
      if (val < m) return bits + (w - 1);
      return bits + (w - 1) + 1;
    }
    int more = x >= mk + a;
    bits += 1;
    if (!more) return bits + b2;
    i++;
    mk += a;
  }
}

// Bits of a unit's parameters against the running references, which it then
// takes (read_lr_unit's order).
HD int unit_bits(int plane, const LrUnit &u, int refW[2][3], int refX[2]) {
  int bits = 0;
  if (u.type == RESTORE_WIENER) {
    for (int pass = 0; pass < 2; pass++)
      for (int j = plane ? 1 : 0; j < 3; j++) {
        bits += subexp_bits(T(Wiener_Taps_Min)[j], T(Wiener_Taps_Max)[j] + 1, T(Wiener_Taps_K)[j], refW[pass][j],
                            u.wiener[pass][j]);
        refW[pass][j] = u.wiener[pass][j];
      }
  } else if (u.type == RESTORE_SGRPROJ) {
    bits += 4;  // SGRPROJ_PARAMS_BITS
    for (int i = 0; i < 2; i++) {
      if (T(Sgr_Params)[u.set][i * 2])
        bits += subexp_bits(T(Sgrproj_Xqd_Min)[i], T(Sgrproj_Xqd_Max)[i] + 1, 4 /* SGRPROJ_PRJ_SUBEXP_K */, refX[i],
                            u.xqd[i]);
      refX[i] = u.xqd[i];
    }
  }
  return bits;
}

HD long long rd(const FrameParams *fp, long long sse, int bits) { return sse * 16 + (long long)fp->lambda * bits; }

// ---- CTA-wide helpers ------------------------------------------------------------------
constexpr int WARPS = THREADS / 32;
struct Shared {
  double acc[12];
  double f[7], g[7];
  long long red[2][WARPS][12];  // a sum's per-warp parts, in turn
  Geom geom;
  Area area;
  int stop;
  uint16_t atab[256];           // self-guided a2 of z (lr_box)
  // k_lr_spec: the unit's candidate cache (Fit::taps / sse / n), kept by thread 0
  int ctaps[CACHE][6];
  long long csse[CACHE];
  int cn, found;
};

// Sum of a 32-bit value over the warp, in 64 bits.
__device__ __forceinline__ long long warp_sum(int v) {
  int hi = __reduce_add_sync(0xffffffffu, v >> 16), lo = __reduce_add_sync(0xffffffffu, v & 0xffff);
  return ((long long)hi << 16) + lo;
}

// Sum of v over the CTA (every thread gets it).
__device__ long long cta_sum(int v, Shared &sh) {
  long long s = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh.red[0][threadIdx.x >> 5][0] = s;
  __syncthreads();
  s = 0;
  for (int w = 0; w < WARPS; w++) s += sh.red[0][w][0];
  return s;
}

// SSE of the unit's CDEF output against the source.
__device__ long long none_sse(const Layout &l, const uint8_t *smem, Shared &sh) {
  const Area &a = sh.area;
  int e = 0;
  for (int k = threadIdx.x; k < a.h * a.w; k += THREADS) {
    int r = quotient(k, a.inv_w), c = k - r * a.w;
    int d = (int)smem[l.tap + (r + 6 * seg_of(a, r) + 3) * l.tap_p + c + 3] - (int)smem[l.src + r * l.src_p + c];
    e += d * d;
  }
  return cta_sum(e, sh);
}

// SSE of the unit filtered with Wiener taps tt (pass 0 vertical j 0..2, pass 1
// horizontal) against the source: flt::lr_wiener's sums and clips. A warp
// takes 16 rows of 32 columns, a lane a column: it keeps the last 7 rows'
// horizontal sums in registers, so a row costs 7 samples read and 8 multiplies
// instead of every 4x4 block filtering 10 rows for 4 (a 64 x 64 unit: 8 tasks,
// one a warp).
constexpr int SSE_ROWS = 16;
__device__ __noinline__ long long wiener_unit_sse(const Layout &l, const uint8_t *smem, const int *tt, Shared &sh) {
  const Area &a = sh.area;
  const int v0 = tt[0], v1 = tt[1], v2 = tt[2], v3 = 128 - 2 * (v0 + v1 + v2);
  const int h0 = tt[3], h1 = tt[4], h2 = tt[5], h3 = 128 - 2 * (h0 + h1 + h2);
  const int offset = 1 << (8 + FILTER_BITS - 3 - 1), limit = (1 << (8 + 1 + FILTER_BITS - 3)) - 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cols = (a.w + 31) >> 5;
  int e = 0, task = 0;
  for (int s = 0; s < a.nseg; s++)
    for (int r0 = a.seg[s]; r0 < a.seg[s + 1]; r0 += SSE_ROWS)
      for (int cg = 0; cg < cols; cg++, task++) {
        if (task % WARPS != warp) continue;
        int x = cg * 32 + lane, r1 = imin(r0 + SSE_ROWS, a.seg[s + 1]);
        if (x >= a.w) continue;
        const uint8_t *t = smem + l.tap + (r0 + 6 * s) * l.tap_p + x;
        const uint8_t *sr = smem + l.src + r0 * l.src_p + x;
        auto hsum = [&](const uint8_t *q) {
          int v = h3 * q[3] + h0 * (q[0] + q[6]) + h1 * (q[1] + q[5]) + h2 * (q[2] + q[4]);
          return clip3(-offset, limit - offset, round2(v, 3));
        };
        int b0 = hsum(t), b1 = hsum(t + l.tap_p), b2 = hsum(t + 2 * l.tap_p), b3 = hsum(t + 3 * l.tap_p),
            b4 = hsum(t + 4 * l.tap_p), b5 = hsum(t + 5 * l.tap_p);
        t += 6 * l.tap_p;
        for (int r = r0; r < r1; r++, t += l.tap_p, sr += l.src_p) {
          int b6 = hsum(t);
          int v = v3 * b3 + v0 * (b0 + b6) + v1 * (b1 + b5) + v2 * (b2 + b4);
          int d = clip3(0, 255, round2(v, 11)) - (int)*sr;
          e += d * d;
          b0 = b1; b1 = b2; b2 = b3; b3 = b4; b4 = b5; b5 = b6;
        }
      }
  return cta_sum(e, sh);
}

HD LrUnit wiener_unit(const int w[2][3]) {
  LrUnit u = {};
  u.type = RESTORE_WIENER;
  for (int p = 0; p < 2; p++)
    for (int j = 0; j < 3; j++) u.wiener[p][j] = w[p][j];
  return u;
}

// wiener_fit (lr_search.c:142-193): four alternating separable least-squares
// solves, then the taps in coded units.
//
// What a sample's 7 values Z[kk] are: the rows (columns) around it filtered by
// the other direction's current taps. A filtered row is the same for the 7
// samples that use it, so each is formed once (hv, in the reference's order of
// additions) instead of once per use. The first solve's taps are the identity:
// its sums are whole numbers, exact in any order, and every thread adds its
// own. The later sums follow the reference's order: one lane per accumulator
// of warp 0 adds a block row's products while the other warps form the next
// row's; that chain of 4,096 dependent double additions a solve bounds the fit.
__device__ void wiener_solve(Shared &sh, int first, int nc, int vertical) {
  double M[3][3] = {{0}}, V[3] = {0}, x[3] = {0, 0, 0};
  for (int a = 0; a < nc; a++) {
    for (int b = 0; b < nc; b++) M[a][b] = sh.acc[a * nc + b];
    V[a] = sh.acc[nc * nc + a];
  }
  for (int a = 0; a < nc; a++) M[a][a] = dadd(M[a][a], 1e-3);
  if (!solve(nc, M, V, x)) {
    sh.stop = 1;
    return;
  }
  double *dst = vertical ? sh.f : sh.g;
  double sum = 0.0;
  for (int k = 0; k < 3; k++) {
    double v = k < first ? 0.0 : x[k - first];
    dst[k] = dst[6 - k] = v;
    sum = dadd(sum, v);
  }
  dst[3] = dsub(1.0, dmul(2.0, sum));
}

__device__ void wiener_fit(const Layout &l, uint8_t *smem, Shared &sh, int out[2][3]) {
  const Area &a = sh.area;
  const int plane = a.plane, first = plane ? 1 : 0, nc = 3 - first, nacc = nc * nc + nc;
  const int lb = plane ? 1 : 2, bwf = 1 << lb;  // block width and height of a 4x4 luma block in this plane
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double *hv = (double *)(smem + l.hv);
  double(*phi)[4] = (double(*)[4])(smem + l.phi);  // two buffers of a block row's samples
  const int rowbuf = bwf * a.w;
  if (tid < 7) sh.f[tid] = sh.g[tid] = tid == 3 ? 1.0 : 0.0;
  if (tid == 0) sh.stop = 0;
  __syncthreads();
  {  // first solve: the taps are the identity, every sum a whole number
    int part[12];
    for (int k = 0; k < 12; k++) part[k] = 0;
    for (int k = tid; k < a.h * a.w; k += THREADS) {
      int r = quotient(k, a.inv_w), c = k - r * a.w;
      const uint8_t *t = smem + l.tap + (r + 6 * seg_of(a, r)) * l.tap_p + c + 3;
      int z3 = t[3 * l.tap_p], ph[4];
      for (int kk = 0; kk < 3; kk++) ph[kk] = (int)t[kk * l.tap_p] + t[(6 - kk) * l.tap_p] - 2 * z3;
      ph[3] = (int)smem[l.src + r * l.src_p + c] - z3;
      for (int i = 0; i < 3; i++)
        for (int j = 0; j < 4; j++) part[i * 4 + j] += ph[i] * ph[j];
    }
    for (int k = 0; k < 12; k++) {
      long long v = warp_sum(part[k]);
      if (lane == 0) sh.red[0][warp][k] = v;
    }
    __syncthreads();
    if (tid < nacc) {
      int i = first + (tid < nc * nc ? tid / nc : tid - nc * nc), j = tid < nc * nc ? first + tid % nc : 3;
      long long v = 0;
      for (int w = 0; w < WARPS; w++) v += sh.red[0][w][i * 4 + j];
      sh.acc[tid] = (double)v;
    }
    __syncthreads();
    if (tid == 0) wiener_solve(sh, first, nc, 1);
    __syncthreads();
  }
  for (int iter = 1; iter < 4 && !sh.stop; iter++) {
    const int vertical = !(iter & 1);
    {  // the filtered rows (vertical solve: hv[tap row][column]) or columns (hv[row][column - 3 .. + 3])
      const double *q = vertical ? sh.g : sh.f;
      const double q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3], q4 = q[4], q5 = q[5], q6 = q[6];
      const int n = vertical ? (a.h + 6 * a.nseg) * a.w : a.h * (a.w + 6);
      for (int k = tid; k < n; k += THREADS) {
        int r = quotient(k, vertical ? a.inv_w : a.inv_w6), c = k - r * (vertical ? a.w : a.w + 6);
        const uint8_t *t = smem + l.tap + (vertical ? r : r + 6 * seg_of(a, r)) * l.tap_p + c;
        const int st = vertical ? 1 : l.tap_p;
        double s = dadd(0.0, dmul(q0, (double)t[0]));
        s = dadd(s, dmul(q1, (double)t[st]));
        s = dadd(s, dmul(q2, (double)t[2 * st]));
        s = dadd(s, dmul(q3, (double)t[3 * st]));
        s = dadd(s, dmul(q4, (double)t[4 * st]));
        s = dadd(s, dmul(q5, (double)t[5 * st]));
        s = dadd(s, dmul(q6, (double)t[6 * st]));
        hv[k] = s;
      }
    }
    __syncthreads();
    const int steps = (a.h + bwf - 1) >> lb;  // block rows
    const int ia = lane < nc * nc ? lane / nc : lane - nc * nc, ib = lane < nc * nc ? lane % nc : 3;
    double acc = 0.0;  // lane L < nacc of warp 0: M[L / nc][L % nc], then V[L - nc * nc]
    for (int step = 0; step <= steps; step++) {
      if (warp > 0 && step < steps) {
        // block row `step` in the reference's order: blocks left to right,
        // each block's rows, each row's samples
        const int i0 = step << lb, h = imin(bwf, a.h - i0), s = seg_of(a, i0);
        double(*ph)[4] = phi + (step & 1) * rowbuf;
        for (int k = tid - 32; k < h * a.w; k += THREADS - 32) {
          int i = quotient(k, a.inv_w), x = k - i * a.w, cb = x >> lb, lbw = imin(bwf, a.w - (cb << lb));
          int o = (cb << lb) * h + i * lbw + x - (cb << lb);
          const double *z = vertical ? hv + (i0 + i + 6 * s) * a.w + x : hv + (i0 + i) * (a.w + 6) + x;
          const int st = vertical ? a.w : 1;
          double z3 = z[3 * st], two = dmul(2.0, z3);
          for (int kk = first; kk < 3; kk++) ph[o][kk - first] = dsub(dadd(z[kk * st], z[(6 - kk) * st]), two);
          ph[o][3] = dsub((double)smem[l.src + (i0 + i) * l.src_p + x], z3);
        }
      } else if (warp == 0 && step > 0 && lane < nacc) {
        const int h = imin(bwf, a.h - ((step - 1) << lb)), n = h * a.w;
        double(*ph)[4] = phi + ((step - 1) & 1) * rowbuf;
        // a batch of products is formed while the one before it is added up
        int k = 0;
        double m[8], nx[8];
        if (n >= 8) {
#pragma unroll
          for (int q = 0; q < 8; q++) m[q] = dmul(ph[q][ia], ph[q][ib]);
        }
        for (; k + 16 <= n; k += 8) {
#pragma unroll
          for (int q = 0; q < 8; q++) nx[q] = dmul(ph[k + 8 + q][ia], ph[k + 8 + q][ib]);
#pragma unroll
          for (int q = 0; q < 8; q++) {
            acc = dadd(acc, m[q]);
            m[q] = nx[q];
          }
        }
        if (n >= 8) {
#pragma unroll
          for (int q = 0; q < 8; q++) acc = dadd(acc, m[q]);
          k += 8;
        }
        for (; k < n; k++) acc = dadd(acc, dmul(ph[k][ia], ph[k][ib]));
      }
      __syncthreads();
    }
    if (tid < nacc) sh.acc[tid] = acc;
    __syncthreads();
    if (tid == 0) wiener_solve(sh, first, nc, vertical);
    __syncthreads();
  }
  for (int pass = 0; pass < 2; pass++) {
    const double *sv = pass == 0 ? sh.f : sh.g;
    for (int j = 0; j < 3; j++) {
      int v = j < first ? 0 : (int)lround_away(dmul(sv[j], 128.0));
      out[pass][j] = j < first ? 0 : imax(T(Wiener_Taps_Min)[j], imin(T(Wiener_Taps_Max)[j], v));
    }
  }
  __syncthreads();
}

// ---- self-guided sets ------------------------------------------------------------------
// flt::lr_box over a whole unit. A position's box sums do not depend on the
// set, so p = n * sum(c^2) - sum(c)^2 and sum(c) of the 5x5 and 3x3 boxes are
// formed once per unit (p1 / b1: 3x3, rows -1 .. rows of each stripe; p2 / b2:
// 5x5, which only odd rows need); a set turns them into (a2, b2) per position,
// and a sample combines its neighbours'. All in 32 bits: a2 <= 256, b2 <=
// 65,088 (255 * 6375 * 164 >> 12), so a sample's sums stay below 2^23.
__device__ void sgr_boxes(const Layout &l, uint8_t *smem, Shared &sh) {
  const Area &a = sh.area;
  const int W2 = a.w + 2;
  uint32_t *p1 = (uint32_t *)(smem + l.p1), *p2 = (uint32_t *)(smem + l.p2);
  uint16_t *b1 = (uint16_t *)(smem + l.b1), *b2 = (uint16_t *)(smem + l.b2);
  for (int k = threadIdx.x; k < (a.h + 2 * a.nseg) * W2; k += THREADS) {
    int r = quotient(k, a.inv_w2), c = k - r * W2, s = 0;
    while (s + 1 < a.nseg && r >= a.seg[s + 1] + 2 * (s + 1)) s++;
    int i = r - 2 * s - a.seg[s] - 1;  // row of the stripe, -1 .. rows
    // the position is tap row (stripe base + i + 3), tap column c + 2
    const uint8_t *t = smem + l.tap + (a.seg[s] + 6 * s + i + 3) * l.tap_p + c + 2;
    int q = 0, m = 0;
    for (int dy = -1; dy <= 1; dy++)
      for (int dx = -1; dx <= 1; dx++) {
        int v = t[dy * l.tap_p + dx];
        q += v * v;
        m += v;
      }
    p1[k] = (uint32_t)(q * 9 - m * m);
    b1[k] = (uint16_t)m;
    if (i & 1) {
      for (int dy = -2; dy <= 2; dy++)
        for (int dx = -2; dx <= 2; dx++) {
          if (dy >= -1 && dy <= 1 && dx >= -1 && dx <= 1) continue;
          int v = t[dy * l.tap_p + dx];
          q += v * v;
          m += v;
        }
      int k2 = (a.seg[s] / 2 + 2 * s + ((i + 1) >> 1)) * W2 + c;
      p2[k2] = (uint32_t)(q * 25 - m * m);
      b2[k2] = (uint16_t)m;
    }
  }
  for (int z = threadIdx.x; z < 256; z += THREADS)
    sh.atab[z] = (uint16_t)(z == 0 ? 1 : z == 255 ? 256 : ((z << SGRPROJ_SGR_BITS) + (z / 2)) / (z + 1));
  __syncthreads();
}

// (a2, b2) of positions 0 .. n - 1 of one box size.
__device__ __forceinline__ void sgr_ab(const uint32_t *p, const uint16_t *b, uint32_t *ab, int n, int boxN, int eps,
                                       const uint16_t *atab) {
  const int n2e = boxN * boxN * eps;
  const unsigned s = ((1 << SGRPROJ_MTABLE_BITS) + n2e / 2) / n2e;
  const unsigned oneOverN = ((1 << SGRPROJ_RECIP_BITS) + (boxN / 2)) / boxN;
  for (int k = threadIdx.x; k < n; k += THREADS) {
    unsigned long long z = ((unsigned long long)p[k] * s + (1u << (SGRPROJ_MTABLE_BITS - 1))) >> SGRPROJ_MTABLE_BITS;
    unsigned a2 = atab[z > 255 ? 255 : (unsigned)z];
    unsigned b2 = ((1u << SGRPROJ_SGR_BITS) - a2) * b[k] * oneOverN;
    ab[k] = a2 | ((b2 + (1u << (SGRPROJ_RECIP_BITS - 1))) >> SGRPROJ_RECIP_BITS) << 16;
  }
}

// sgr_fit (lr_search.c:196-240) and the SSE of the fitted set, for sets s0 ..
// s1 - 1. The fit's sums are whole numbers and exact in 64 bits; the closing
// double arithmetic follows the reference's operations. With weights w0, w2
// and w1 = 128 - w0 - w2 the projection w1 u + w0 F0 + w2 F1 is 128 u +
// w0 (F0 - u) + w2 (F1 - u): the differences the fit forms are kept (fd) and
// give the SSE without filtering again.
__device__ void sgr_sets(const Layout &l, uint8_t *smem, int s0, int s1, Fit &F, Shared &sh) {
  const Area &a = sh.area;
  const int W2 = a.w + 2, n1 = (a.h + 2 * a.nseg) * W2, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t *p1 = (const uint32_t *)(smem + l.p1), *p2 = (const uint32_t *)(smem + l.p2);
  const uint16_t *b1 = (const uint16_t *)(smem + l.b1), *b2 = (const uint16_t *)(smem + l.b2);
  uint32_t *ab1 = (uint32_t *)(smem + l.ab1), *ab2 = (uint32_t *)(smem + l.ab2), *fd = (uint32_t *)(smem + l.fd);
  sgr_boxes(l, smem, sh);
  const int n2 = a.nseg ? (a.seg[a.nseg - 1] / 2 + 2 * (a.nseg - 1) + (a.h - a.seg[a.nseg - 1] + 1) / 2 + 1) * W2 : 0;
  for (int set = s0; set < s1; set++) {
    const int r0 = T(Sgr_Params)[set][0], r1 = T(Sgr_Params)[set][2];
    // the first filter's box is 5x5 and the second's 3x3 in every set that has them
    if (r0) sgr_ab(p2, b2, ab2, n2, 25, T(Sgr_Params)[set][1], sh.atab);
    if (r1) sgr_ab(p1, b1, ab1, n1, 9, T(Sgr_Params)[set][3], sh.atab);
    __syncthreads();
    int h00 = 0, h01 = 0, h11 = 0, c0 = 0, c1 = 0;
    for (int k = tid; k < a.h * a.w; k += THREADS) {
      int r = quotient(k, a.inv_w), x = k - r * a.w, s = seg_of(a, r), i = r - a.seg[s];
      int own = smem[l.tap + (r + 6 * s + 3) * l.tap_p + x + 3];
      int u = own << SGRPROJ_RST_BITS, sd = ((int)smem[l.src + r * l.src_p + x] << SGRPROJ_RST_BITS) - u;
      int d0 = 0, d1 = 0;
      if (r0) {
        // odd rows carry the sums: an odd row uses its own, an even row the two around it
        const uint32_t *q = ab2 + (a.seg[s] / 2 + 2 * s + ((i + 1) >> 1)) * W2 + x;
        unsigned l0 = q[0], m0 = q[1], e0 = q[2];
        unsigned A = 6 * (m0 & 0xffff) + 5 * ((l0 & 0xffff) + (e0 & 0xffff)), B = 6 * (m0 >> 16) + 5 * ((l0 >> 16) + (e0 >> 16));
        int sh0 = SGRPROJ_SGR_BITS + 4 - SGRPROJ_RST_BITS;
        if (!(i & 1)) {
          unsigned l1 = q[W2], m1 = q[W2 + 1], e1 = q[W2 + 2];
          A += 6 * (m1 & 0xffff) + 5 * ((l1 & 0xffff) + (e1 & 0xffff));
          B += 6 * (m1 >> 16) + 5 * ((l1 >> 16) + (e1 >> 16));
          sh0++;
        }
        d0 = (int)((A * own + B + (1u << (sh0 - 1))) >> sh0) - u;
      }
      if (r1) {
        const uint32_t *q = ab1 + (r + 2 * s) * W2 + x;
        unsigned A = 0, B = 0;
#pragma unroll
        for (int dy = 0; dy < 3; dy++)
#pragma unroll
          for (int dx = 0; dx < 3; dx++) {
            unsigned v = q[dy * W2 + dx], wgt = dy == 1 || dx == 1 ? 4 : 3;
            A += wgt * (v & 0xffff);
            B += wgt * (v >> 16);
          }
        constexpr int sh1 = SGRPROJ_SGR_BITS + 5 - SGRPROJ_RST_BITS;
        d1 = (int)((A * own + B + (1u << (sh1 - 1))) >> sh1) - u;
      }
      fd[k] = (uint32_t)(d0 & 0xffff) | (uint32_t)d1 << 16;
      h00 += d0 * d0;
      h01 += d0 * d1;
      h11 += d1 * d1;
      c0 += d0 * sd;
      c1 += d1 * sd;
    }
    const int par = set & 1;
    {
      long long v0 = warp_sum(h00), v1 = warp_sum(h01), v2 = warp_sum(h11), v3 = warp_sum(c0), v4 = warp_sum(c1);
      if (lane == 0) {
        long long *o = sh.red[par][warp];
        o[0] = v0; o[1] = v1; o[2] = v2; o[3] = v3; o[4] = v4;
      }
    }
    __syncthreads();
    long long sum[5] = {0, 0, 0, 0, 0};
    for (int w = 0; w < WARPS; w++)
      for (int k = 0; k < 5; k++) sum[k] += sh.red[par][w][k];
    double H00 = (double)sum[0], H01 = (double)sum[1], H11 = (double)sum[2], C0 = (double)sum[3], C1 = (double)sum[4];
    double fa = 0.0, fb = 0.0;
    if (r0 && r1) {
      double det = dsub(dmul(H00, H11), dmul(H01, H01));
      if (fabs(det) > 1e-9) {
        fa = ddiv(dsub(dmul(C0, H11), dmul(C1, H01)), det);
        fb = ddiv(dsub(dmul(C1, H00), dmul(C0, H01)), det);
      }
    } else if (r0) {
      if (H00 > 0) fa = ddiv(C0, H00);
    } else if (r1) {
      if (H11 > 0) fb = ddiv(C1, H11);
    }
    int w0 = (int)lround_away(dmul(fa, (double)(1 << SGRPROJ_PRJ_BITS)));
    int w2 = (int)lround_away(dmul(fb, (double)(1 << SGRPROJ_PRJ_BITS)));
    if (!r0) w0 = 0;
    const int x0 = imax(T(Sgrproj_Xqd_Min)[0], imin(T(Sgrproj_Xqd_Max)[0], w0));
    const int x1 = imax(T(Sgrproj_Xqd_Min)[1],
                        imin(T(Sgrproj_Xqd_Max)[1], (1 << SGRPROJ_PRJ_BITS) - x0 - (r1 ? w2 : 0)));
    const int x2 = (1 << SGRPROJ_PRJ_BITS) - x0 - x1;
    int e = 0;
    for (int k = tid; k < a.h * a.w; k += THREADS) {
      int r = quotient(k, a.inv_w), x = k - r * a.w, s = seg_of(a, r);
      int u = (int)smem[l.tap + (r + 6 * s + 3) * l.tap_p + x + 3] << SGRPROJ_RST_BITS;
      int d0 = (int)(int16_t)(fd[k] & 0xffff), d1 = (int)fd[k] >> 16;
      int v = (u << SGRPROJ_PRJ_BITS) + x0 * d0 + x2 * d1;
      int d = clip3(0, 255, round2(v, SGRPROJ_RST_BITS + SGRPROJ_PRJ_BITS)) - (int)smem[l.src + r * l.src_p + x];
      e += d * d;
    }
    long long ew = warp_sum(e);
    if (lane == 0) sh.red[par][warp][5] = ew;
    if (tid == 0) {
      F.xqd[set][0] = x0;
      F.xqd[set][1] = x1;
    }
    // the next set's barriers order these parts; the one after it writes this
    // buffer again only after this set's SSE has been read
    __syncthreads();
    if (tid == 0) {
      long long t = 0;
      for (int w = 0; w < WARPS; w++) t += sh.red[par][w][5];
      F.sgr_sse[set] = t;
    }
  }
}

HD void taps_of(const LrUnit &u, int *t) {
  for (int p = 0; p < 2; p++)
    for (int j = 0; j < 3; j++) t[p * 3 + j] = u.wiener[p][j];
}

// The unit `gu` of LRUNITS: its plane, place and area, staged (the whole CTA).
__device__ void load_unit(const FrameParams *fp, int gu, const uint8_t *cdef, const uint8_t *dbk, const uint8_t *src,
                          const Layout &l, uint8_t *smem, Shared &sh) {
  if (threadIdx.x == 0) {
    int plane = 2;
    while (plane > 0 && gu < fp->lr_unit_off[plane]) plane--;
    const int u = gu - fp->lr_unit_off[plane];
    unit_geom(fp, plane, u / fp->lr_unit_cols[plane], u % fp->lr_unit_cols[plane], &sh.geom);
    unit_area(fp, sh.geom, &sh.area);
  }
  __syncthreads();
  stage_unit(fp, sh.area, cdef, dbk, src, l, smem);
}

// First pass, all planes at once: CTA (unit, part). Part 0 fits the Wiener
// filter and takes its SSEs (latency: the fit's ordered sums), parts 1 and 2
// take half of the self-guided sets each, so a small frame's units spread over
// three times the SMs. With one CTA per unit, a 4x4 block a thread and every
// block's taps clamped and box sums formed anew, the pass took 7.06 ms for a
// 1280x720 frame's units and 42.8 ms at 3840x2160; this form takes 0.81 and
// 3.97 ms.
constexpr int FIT_PARTS = 3;
__global__ void __launch_bounds__(THREADS, 2) k_lr_fit(const FrameParams *fp, const uint8_t *cdef, const uint8_t *dbk,
                                                      const uint8_t *src, Fit *fits, Dims dims) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ Shared sh;
  const Layout l = layout_of(dims);
  const int gu = blockIdx.x / FIT_PARTS, part = blockIdx.x % FIT_PARTS;
  load_unit(fp, gu, cdef, dbk, src, l, smem, sh);
  Fit &F = fits[gu];
  if (part > 0) {
    sgr_sets(l, smem, part == 1 ? 0 : 8, part == 1 ? 8 : 16, F, sh);
    return;
  }
  const int plane = sh.area.plane;
  long long sseNone = none_sse(l, smem, sh);
  int w[2][3];
  wiener_fit(l, smem, sh, w);
  // the fitted filter and its single-tap neighbours, in the refinement's order
  int n = 0, tt[6];
  LrUnit base = wiener_unit(w);
  taps_of(base, tt);
  long long sseW = wiener_unit_sse(l, smem, tt, sh);
  if (threadIdx.x == 0) {
    taps_of(base, F.taps[n]);
    F.sse[n] = sseW;
  }
  n++;
  for (int pass = 0; pass < 2; pass++)
    for (int j = plane ? 1 : 0; j < 3; j++)
      for (int d = -1; d <= 1; d += 2) {
        LrUnit t = base;
        t.wiener[pass][j] += d;
        if (t.wiener[pass][j] < T(Wiener_Taps_Min)[j] || t.wiener[pass][j] > T(Wiener_Taps_Max)[j]) continue;
        taps_of(t, tt);
        long long sse = wiener_unit_sse(l, smem, tt, sh);
        if (threadIdx.x == 0) {
          taps_of(t, F.taps[n]);
          F.sse[n] = sse;
        }
        n++;
      }
  if (threadIdx.x == 0) {
    F.sse_none = sseNone;
    F.n = F.n0 = n;
    for (int p = 0; p < 2; p++)
      for (int j = 0; j < 3; j++) F.w[p][j] = w[p][j];
  }
}

// Index of the cache entry holding taps tt (entries are distinct), or -1:
// thread i compares entry i (the whole CTA).
__device__ int cache_find(const int (*taps)[6], int n, const int *tt, Shared &sh) {
  if (threadIdx.x == 0) sh.found = -1;
  __syncthreads();
  int i = threadIdx.x;
  if (i < n) {
    bool eq = true;
    for (int k = 0; k < 6; k++) eq = eq && taps[i][k] == tt[k];
    if (eq) sh.found = i;
  }
  __syncthreads();
  int f = sh.found;
  __syncthreads();
  return f;
}

// Speculative refinement, one CTA per unit, after k_lr_fit: the Wiener
// refinement of lr_select (lr_search.c:296-318) replayed for the unit under
// guessed running references, computing and caching the SSE of every
// candidate the cache does not hold yet. An SSE depends on the candidate
// filter and the unit's samples only, never on the references, so a cached
// value is exactly what the serial choice would compute; the references only
// decide which candidates the refinement visits. The guesses: the default
// references (exact for a plane's first unit) and the fitted filter of each
// of the two previous units (the true reference is usually the refined
// filter of a recent unit). k_lr_select then finds most of its candidates
// here and computes only the rest on the spot.
__device__ void spec_path(const FrameParams *fp, int plane, const Layout &l, const uint8_t *smem, const int fitted[2][3],
                          const int ref[2][3], int room, Shared &sh) {
  LrUnit w = wiener_unit(fitted);
  int tw[2][3], tx[2] = {0, 0};
  memcpy(tw, ref, sizeof tw);
  long long wc = rd(fp, sh.csse[0], 2 + unit_bits(plane, w, tw, tx));
  for (int pass = 0; pass < 2; pass++)
    for (int j = plane ? 1 : 0; j < 3; j++)
      for (int d = -1; d <= 1; d += 2) {
        LrUnit t = w;
        t.wiener[pass][j] += d;
        if (t.wiener[pass][j] < T(Wiener_Taps_Min)[j] || t.wiener[pass][j] > T(Wiener_Taps_Max)[j]) continue;
        int tt[6];
        taps_of(t, tt);
        int n = sh.cn;
        int f = cache_find(sh.ctaps, n, tt, sh);
        long long sse = f >= 0 ? sh.csse[f] : -1;
        if (sse < 0) {
          if (n >= room) return;  // full: the serial choice computes the rest
          sse = wiener_unit_sse(l, smem, tt, sh);  // the whole CTA; every thread gets the sum
          if (threadIdx.x == 0) {
            for (int k = 0; k < 6; k++) sh.ctaps[n][k] = tt[k];
            sh.csse[n] = sse;
            sh.cn = n + 1;
          }
          __syncthreads();
        }
        memcpy(tw, ref, sizeof tw);
        long long tc = rd(fp, sse, 2 + unit_bits(plane, t, tw, tx));
        if (tc < wc) {
          wc = tc;
          w = t;
        }
      }
}

// room: cached candidates a unit keeps (CACHE unless a test lowers it)
__global__ void __launch_bounds__(THREADS) k_lr_spec(const FrameParams *fp, const uint8_t *cdef, const uint8_t *dbk,
                                                    const uint8_t *src, Fit *fits, Dims dims, int room) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ Shared sh;
  const Layout l = layout_of(dims);
  const int gu = blockIdx.x;
  Fit &F = fits[gu];
  if (threadIdx.x == 0) sh.cn = F.n;
  for (int i = threadIdx.x; i < F.n * 6; i += THREADS) sh.ctaps[i / 6][i % 6] = F.taps[i / 6][i % 6];
  for (int i = threadIdx.x; i < F.n; i += THREADS) sh.csse[i] = F.sse[i];
  load_unit(fp, gu, cdef, dbk, src, l, smem, sh);
  const int plane = sh.area.plane, u = gu - fp->lr_unit_off[plane];
  const int n0 = sh.cn;
  int fitted[2][3], ref[2][3];
  for (int pass = 0; pass < 2; pass++)
    for (int j = 0; j < 3; j++) fitted[pass][j] = F.w[pass][j];
  for (int q = 0; q < 3 && q <= u; q++) {
    for (int pass = 0; pass < 2; pass++)
      for (int j = 0; j < 3; j++) ref[pass][j] = q == 0 ? T(Wiener_Taps_Mid)[j] : fits[gu - q].w[pass][j];
    spec_path(fp, plane, l, smem, fitted, ref, room, sh);
  }
  __syncthreads();
  const int n1 = sh.cn;
  for (int i = n0 * 6 + threadIdx.x; i < n1 * 6; i += THREADS) F.taps[i / 6][i % 6] = sh.ctaps[i / 6][i % 6];
  for (int i = n0 + threadIdx.x; i < n1; i += THREADS) F.sse[i] = sh.csse[i];
  if (threadIdx.x == 0) F.n = n1;
}

// ---- the choice ----------------------------------------------------------------------------
// A unit's choice depends on the units before it only through the running
// references: the taps of the last Wiener unit and the weights of the last
// self-guided one. lr_select's serial scan (lr_search.c:276-355) is therefore
// the one assignment in which every unit is chosen with the references its
// predecessors leave, and it is found by guessing: k_lr_choose chooses every
// unit at once, a warp each, first with its predecessor's fitted filter for
// reference, then with the references the first choices leave; k_lr_select
// (one CTA per plane) chooses again the units whose references differ from
// those they were chosen with, until there are none. Unit by unit from the
// first, such an assignment equals the scan's; nearly every unit stands after
// the second guess. (A warp's scan of the units in order took 3.9 us a unit:
// 7.9 ms for a 3840x2160 frame.)
//
// Within a unit: a filter's rate is the sum of its taps' (unit_bits), the
// refinement moves one tap at a time and a tap by at most one, so 18 lanes
// code each tap's three values once and a candidate's rate is its
// predecessor's with one term exchanged; 16 lanes code the self-guided sets. A
// candidate is 6 two-bit steps from the fitted filter: lanes compare the
// cached candidates' codes at once.
constexpr int FIT_WORDS = (int)(sizeof(Fit) / 4);
static_assert(sizeof(Fit) % 4 == 0 && CACHE <= 64, "two cached candidates a lane");
constexpr int UNUSED_REF = 0x7fffffff;  // Fit::used[0]: choose again

// Chooses unit u of the plane (LRUNITS record `unit`) under the references
// ref[0..5] (taps) and ref[6], ref[7] (weights), by one warp; F: the unit's
// record in shared memory. False if a candidate's SSE is not cached: its taps
// are then in miss (lane c: tap c), and the unit is not written.
__device__ bool choose_unit(const FrameParams *fp, int plane, int u, const Fit &F, const int *ref, int lrTest, LrUnit *unit, int *miss) {
  const int lane = threadIdx.x & 31, first = plane ? 1 : 0;
  const long long lambda = fp->lambda;
  const int *fw = &F.w[0][0];
  // lane 3 c + d + 1, c = 3 pass + j: tap c moved by d (a value out of range is never a candidate)
  const int myC = imin(lane / 3, 5), myJ = myC % 3;
  const int tapMin = T(Wiener_Taps_Min)[myJ], tapMax = T(Wiener_Taps_Max)[myJ];
  const int v = fw[myC] + lane % 3 - 1;
  const bool ok = lane < 18 && myJ >= first && v >= tapMin && v <= tapMax;
  const int tb = ok ? subexp_bits(tapMin, tapMax + 1, T(Wiener_Taps_K)[myJ], ref[myC], v) : 0;
  const unsigned okMask = __ballot_sync(0xffffffffu, ok);
  // rate of this lane's self-guided set
  const int set = lane & 15;
  int sb = 2 + 4;
  if (T(Sgr_Params)[set][0]) sb += subexp_bits(T(Sgrproj_Xqd_Min)[0], T(Sgrproj_Xqd_Max)[0] + 1, 4, ref[6], F.xqd[set][0]);
  if (T(Sgr_Params)[set][2]) sb += subexp_bits(T(Sgrproj_Xqd_Min)[1], T(Sgrproj_Xqd_Max)[1] + 1, 4, ref[7], F.xqd[set][1]);
  // this lane's cached candidates as steps from the fitted filter: (d + 1) << 2 c
  unsigned code[2];
  long long csse[2];
#pragma unroll
  for (int q = 0; q < 2; q++) {
    int i = lane + 32 * q;
    code[q] = ~0u;
    csse[q] = 0;
    if (i < F.n) {
      unsigned cd = 0;
      for (int c = 0; c < 6; c++) cd |= (unsigned)((F.taps[i][c] - fw[c] + 1) & 3) << (2 * c);
      code[q] = cd;
      csse[q] = F.sse[i];
    }
  }
  // the refinement (lr_search.c:296-318)
  int bits = 2;
  for (int c = 0; c < 6; c++)
    if (c % 3 >= first) bits += __shfl_sync(0xffffffffu, tb, 3 * c + 1);
  unsigned cur = 0x555;
  long long wc = F.sse[0] * 16 + lambda * bits;
  for (int c = 0; c < 6; c++) {
    if (c % 3 < first) continue;
    for (int d = -1; d <= 1; d += 2) {
      int at = (int)(cur >> (2 * c)) & 3, to = at + d;  // d + 1 of the tap now and moved
      if (!((okMask >> (3 * c + to)) & 1)) continue;
      unsigned want = (cur & ~(3u << (2 * c))) | (unsigned)to << (2 * c);
      int tbits = bits - __shfl_sync(0xffffffffu, tb, 3 * c + at) + __shfl_sync(0xffffffffu, tb, 3 * c + to);
      unsigned m0 = __ballot_sync(0xffffffffu, code[0] == want), m1 = __ballot_sync(0xffffffffu, code[1] == want);
      if (!(m0 | m1)) {
        if (lane < 6) miss[lane] = fw[lane] + ((int)(want >> (2 * lane)) & 3) - 1;
        __syncwarp();
        return false;
      }
      long long sse = __shfl_sync(0xffffffffu, m0 ? csse[0] : csse[1], __ffs(m0 ? m0 : m1) - 1);
      long long tc = sse * 16 + lambda * tbits;
      if (tc < wc) {
        wc = tc;
        cur = want;
        bits = tbits;
      }
    }
  }
  int type = RESTORE_NONE;
  long long bestCost = rd(fp, F.sse_none, 1);
  if (wc < bestCost) {
    bestCost = wc;
    type = RESTORE_WIENER;
  }
  // first least of the sets' costs (with lrTest on odd units: of their SSEs)
  const bool testSgr = lrTest && (u & 1);
  long long sc = testSgr ? F.sgr_sse[set] : F.sgr_sse[set] * 16 + lambda * sb;
  int si = set;
  for (int o = 8; o; o >>= 1) {
    long long oc = __shfl_xor_sync(0xffffffffu, sc, o);
    int oi = __shfl_xor_sync(0xffffffffu, si, o);
    if (oc < sc || (oc == sc && oi < si)) {
      sc = oc;
      si = oi;
    }
  }
  if (testSgr || sc < bestCost) type = RESTORE_SGRPROJ;
  if (lrTest && !(u & 1)) type = RESTORE_WIENER;  // Wiener on even units, the least SSE's set on odd ones
  // the record: type, set, xqd[2], wiener[2][3], pad[2]
  const int tapv = lane < 6 ? fw[lane] + ((int)(cur >> (2 * lane)) & 3) - 1 : 0;
  const int wv = __shfl_sync(0xffffffffu, tapv, lane >= 4 && lane < 10 ? lane - 4 : 0);
  int o = 0;
  if (lane == 0) o = type;
  else if (type == RESTORE_SGRPROJ) o = lane == 1 ? si : lane == 2 ? F.xqd[si][0] : lane == 3 ? F.xqd[si][1] : 0;
  else if (type == RESTORE_WIENER && lane >= 4 && lane < 10) o = wv;
  if (lane < (int)(sizeof(LrUnit) / 4)) ((int *)unit)[lane] = o;
  return true;
}

struct ChooseMem {
  Fit fit;
  int ref[8], miss[6];
};
__device__ __forceinline__ void load_fit(const Fit *F, Fit &to) {
  for (int k = threadIdx.x & 31; k < FIT_WORDS; k += 32) ((int *)&to)[k] = __ldcg((const int *)F + k);
}
__device__ __forceinline__ int default_ref(int k) { return k < 6 ? T(Wiener_Taps_Mid)[k % 3] : T(Sgrproj_Xqd_Mid)[k - 6]; }

// The references that the units before u leave, lane k < 8 the k-th (a warp):
// the last Wiener unit's taps, the last self-guided unit's weights.
__device__ int running_ref(const LrUnit *units, int u, int first) {
  const int lane = threadIdx.x & 31;
  int wi = -1, si = -1;
  for (int e = u; e > 0 && (wi < 0 || si < 0); e -= 32) {
    int k = e - 1 - lane, t = k >= 0 ? __ldcg(&units[k].type) : RESTORE_NONE;
    unsigned mw = __ballot_sync(0xffffffffu, t == RESTORE_WIENER), ms = __ballot_sync(0xffffffffu, t == RESTORE_SGRPROJ);
    if (wi < 0 && mw) wi = e - __ffs(mw);
    if (si < 0 && ms) si = e - __ffs(ms);
  }
  int r = lane < 8 ? default_ref(lane) : 0;
  if (wi >= 0 && lane < 6 && lane % 3 >= first) r = __ldcg(&units[wi].wiener[0][0] + lane);
  if (si >= 0 && lane >= 6 && lane < 8) r = __ldcg(&units[si].xqd[0] + lane - 6);
  return r;
}

// A guess for every unit at once, a warp each. pass 0: the references are the
// previous unit's fitted filter and the default weights; pass 1: what the
// units before it chose in pass 0 (or, for one being chosen again meanwhile,
// in this pass: a guess all the same, recorded as used).
__global__ void __launch_bounds__(THREADS) k_lr_choose(const FrameParams *fp, Fit *fits, LrUnit *units, int lrTest, int n, int pass) {
  __shared__ ChooseMem mem[WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gu = blockIdx.x * WARPS + warp;
  if (gu >= n) return;
  ChooseMem &m = mem[warp];
  int plane = 2;
  while (plane > 0 && gu < fp->lr_unit_off[plane]) plane--;
  const int off = fp->lr_unit_off[plane], u = gu - off;
  load_fit(fits + gu, m.fit);
  int r = lane < 8 ? default_ref(lane) : 0;
  if (pass == 0) {
    if (u > 0 && lane < 6 && lane % 3 >= (plane ? 1 : 0)) r = __ldcg(&fits[gu - 1].w[0][0] + lane);
  } else {
    r = running_ref(units + off, u, plane ? 1 : 0);
  }
  if (lane < 8) m.ref[lane] = r;
  __syncwarp();
  if (pass == 1) {  // chosen with these references already
    int same = lane < 8 ? m.fit.used[lane] == r : 1;
    if (__all_sync(0xffffffffu, same)) return;
  }
  bool done = choose_unit(fp, plane, u, m.fit, m.ref, lrTest, units + gu, m.miss);
  if (!done && lane < (int)(sizeof(LrUnit) / 4) && pass == 0) ((int *)(units + gu))[lane] = 0;
  if (lane < 8) fits[gu].used[lane] = done ? r : UNUSED_REF;
}

// The units whose references differ from those they were chosen with, until
// there are none: in rounds, all of them at once, a warp each, while no
// candidate's SSE is missing. A missing one is filtered by the whole CTA, and
// only for a unit whose references are settled (everything before it stands):
// from the first miss on the first unit that differs and those after it are
// taken in order, a warp alone between two misses, up to a run of units that
// stand. Filtering misses for every unit of a round as well, under references
// that the next round changed again, took 164 ms a 3840x2160 frame at
// quantizer 255, where a scan of all units had left the whole search at 140;
// now 55 ms (quantizer 150: 34 -> 23; 20, without misses: 5.3 as before).
// listRoom, room: units a round chooses again, cached candidates a unit keeps
// (LIST and CACHE unless a test lowers them; at least 1 and MIN_CACHE).
constexpr int ROUNDS = 4;     // rounds before the units are taken in order in any case
constexpr int STANDING = 16;  // standing units after which the whole plane is looked at again
__global__ void __launch_bounds__(THREADS) k_lr_select(FrameParams *fp, const uint8_t *cdef, const uint8_t *dbk,
                                                      const uint8_t *src, Fit *fits, LrUnit *units,
                                                      int lrTest, int *lrTypes, Dims dims, int listRoom, int room) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ Shared sh;
  __shared__ ChooseMem mem[WARPS];
  __shared__ int lastW[THREADS], lastS[THREADS], todo, any, lowest, missed, job;
  __shared__ int list[LIST];
  const Layout l = layout_of(dims);
  const int plane = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, first = plane ? 1 : 0;
  const int nUnits = fp->lr_unit_rows[plane] * fp->lr_unit_cols[plane], off = fp->lr_unit_off[plane];
  const int per = (nUnits + THREADS - 1) / THREADS, u0 = imin(nUnits, tid * per), u1 = imin(nUnits, u0 + per);
  if (tid == 0) missed = 0;
  for (int round = 0;; round++) {
    // each thread's run of units: the last Wiener and self-guided unit before
    // it, then every unit's references against those it was chosen with
    if (tid == 0) {
      todo = any = 0;
      lowest = nUnits;
    }
    int w = -1, g = -1;
    for (int u = u0; u < u1; u++) {
      int t = __ldcg(&units[off + u].type);
      if (t == RESTORE_WIENER) w = u;
      else if (t == RESTORE_SGRPROJ) g = u;
    }
    lastW[tid] = w;
    lastS[tid] = g;
    __syncthreads();
    for (int o = 1; o < THREADS; o <<= 1) {
      int a = tid >= o ? lastW[tid - o] : -1, b = tid >= o ? lastS[tid - o] : -1;
      __syncthreads();
      lastW[tid] = imax(lastW[tid], a);
      lastS[tid] = imax(lastS[tid], b);
      __syncthreads();
    }
    if (w >= 0 || g >= 0) any = 1;
    w = tid ? lastW[tid - 1] : -1;
    g = tid ? lastS[tid - 1] : -1;
    for (int u = u0; u < u1; u++) {
      const Fit &F = fits[off + u];
      bool same = true;
      for (int k = 0; k < 8; k++) {
        int r = default_ref(k);
        if (k < 6 && w >= 0 && k % 3 >= first) r = __ldcg(&units[off + w].wiener[0][0] + k);
        if (k >= 6 && g >= 0) r = __ldcg(&units[off + g].xqd[0] + k - 6);
        same = same && r == __ldcg(F.used + k);
      }
      if (!same) {  // what the list has no room for is found again in the next round
        atomicMin(&lowest, u);
        int slot = atomicAdd(&todo, 1);
        if (slot < listRoom) list[slot] = u;
      }
      int t = __ldcg(&units[off + u].type);
      if (t == RESTORE_WIENER) w = u;
      else if (t == RESTORE_SGRPROJ) g = u;
    }
    __syncthreads();
    const int n = imin(todo, listRoom), low = lowest;
    if (n == 0) break;
    if (missed || round >= ROUNDS) {
      // in order from the first unit that differs
      int u = low, r = 0, stood = 0, staged = -1;
      bool again = false;  // unit u, its record loaded, after a miss
      if (warp == 0) r = running_ref(units + off, u, first);
      for (;;) {
        if (warp == 0) {
          ChooseMem &m = mem[0];
          int miss = -1;
          for (; u < nUnits && stood < STANDING; u++, again = false) {
            if (!again) {
              bool same = lane >= 8 || __ldcg(&fits[off + u].used[lane & 7]) == r;
              stood = __all_sync(0xffffffffu, same) ? stood + 1 : 0;
              if (stood == 0) {
                load_fit(fits + off + u, m.fit);
                if (lane < 8) m.ref[lane] = r;
                __syncwarp();
              }
            }
            if (stood == 0) {
              if (!choose_unit(fp, plane, u, m.fit, m.ref, lrTest, units + off + u, m.miss)) {
                miss = u;
                again = true;
                break;
              }
              if (lane < 8) fits[off + u].used[lane] = r;
              __syncwarp();
            }
            const int t = __ldcg(&units[off + u].type);
            if (t == RESTORE_WIENER && lane < 6 && lane % 3 >= first) r = __ldcg(&units[off + u].wiener[0][0] + lane);
            if (t == RESTORE_SGRPROJ && lane >= 6 && lane < 8) r = __ldcg(&units[off + u].xqd[0] + lane - 6);
          }
          if (lane == 0) job = miss;
        }
        __syncthreads();
        const int ju = job;
        if (ju < 0) break;
        if (staged != ju) load_unit(fp, off + ju, cdef, dbk, src, l, smem, sh);
        staged = ju;
        int tt[6];
        for (int c = 0; c < 6; c++) tt[c] = mem[0].miss[c];
        long long sse = wiener_unit_sse(l, smem, tt, sh);
        if (tid == 0) {
          Fit &F = mem[0].fit;
          // a full cache keeps the first pass's candidates: a path under
          // settled references needs at most 12 more
          int at = F.n < room ? F.n : F.n0;
          for (int c = 0; c < 6; c++) F.taps[at][c] = tt[c];
          F.sse[at] = sse;
          F.n = at + 1;
        }
        __syncthreads();
      }
      continue;
    }
    // the first of them is always among them, once: it is chosen for good, so the rounds end
    if (tid == 0 && todo > listRoom) {
      for (int k = 1; k < n; k++)
        if (list[k] == low) list[k] = list[0];
      list[0] = low;
    }
    __syncthreads();
    for (int k = warp; k < n; k += WARPS) {
      const int u = list[k];
      ChooseMem &m = mem[warp];
      load_fit(fits + off + u, m.fit);
      const int r = running_ref(units + off, u, first);
      if (lane < 8) m.ref[lane] = r;
      __syncwarp();
      bool done = choose_unit(fp, plane, u, m.fit, m.ref, lrTest, units + off + u, m.miss);
      if (lane < 8) fits[off + u].used[lane] = done ? r : UNUSED_REF;
      if (!done && lane == 0) missed = 1;
      __syncwarp();
    }
    __syncthreads();
  }
  if (tid == 0) fp->lr_type[plane] = lrTypes[plane] = any ? RESTORE_SWITCHABLE : RESTORE_NONE;
}

}  // namespace lrs
