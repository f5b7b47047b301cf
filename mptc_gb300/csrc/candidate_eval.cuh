// Evaluation of a candidate index word on a block (the refit, snap, validity
// and error of DXTImage::Reencode, codec/dxt_image.cpp:258-349) and the
// staging of the block it needs.
#pragma once
#include <cstdint>

#include "status_bits.cuh"

namespace mptc {

constexpr uint32_t kFull = 0xffffffffu;
constexpr int kInvalid = 0x7fffffff;  // invalid candidate / no selection (INT_MAX)


// Staging of the block being searched (one per warp in the inter search, one
// per CTA in the intra search).
//
// The refit accumulates, per pixel i and channel c, ax += px*a and bx += px*b
// with (a, b) = ((3-order)/3, order/3), order = {0,3,1,2}[index]. For the four
// index values the products are exactly (px, 0), (0, px), (2q, q), (q, 2q)
// with q = fl(px * fl(1/3)) (fl(2/3) = 2 fl(1/3), and doubling is exact), so
// the block keeps them as a table ab[i][index] = {A.xyz, B.xyz} and a
// candidate's refit becomes one lookup and six adds per pixel.
//
// Layout ab[pixel][part][index] (float2): part 0 = (A_r, A_g), 1 = (A_b, B_r),
// 2 = (B_g, B_b). The four index variants of one (pixel, part) are adjacent,
// so the lanes of a warp, whatever their indices, read distinct banks.
struct __align__(16) BlockTab {
  float2 ab[16][3][4];
  uint32_t pg[3][4];    // channel c bytes of pixels 4g .. 4g+3 (for dp4a)
};

// The twelve channel-group words of the staged block, held in registers.
struct PixelGroups {
  uint32_t w[3][4];
};

__device__ __forceinline__ PixelGroups load_groups(const BlockTab &t) {
  PixelGroups g;
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int k = 0; k < 4; ++k) g.w[c][k] = t.pg[c][k];
  return g;
}

// Per-candidate weight sums of the refit (they depend on the index word only).
struct WeightSums {
  float asq, bsq, ab, f;  // f = 1 / (asq*bsq - ab*ab)
};

// ToFiveBits / ToSixBits (codec/dxt_image.cpp:72-121) as 256-entry tables,
// built per CTA in shared memory: value -> snapped 8-bit value.
__device__ __forceinline__ uint8_t snap_value(uint32_t x, uint32_t keep, uint32_t step, uint32_t sh) {
  uint32_t base = x & keep;
  uint32_t high = (base == 255u) ? base : base + step;
  uint32_t low = (base == 0u) ? base : base - step;
  base = (base | (base >> sh)) & 0xFF;
  high = (high | (high >> sh)) & 0xFF;
  low = (low | (low >> sh)) & 0xFF;
  const uint32_t db = x > base ? x - base : base - x;
  const uint32_t dh = x > high ? x - high : high - x;
  const uint32_t dl = x > low ? x - low : low - x;
  if (db <= dh) return (uint8_t)(db < dl ? base : low);
  return (uint8_t)high;
}

__device__ __forceinline__ void build_snap_tables(uint8_t *snap5, uint8_t *snap6) {
  for (int t = threadIdx.x; t < 256; t += blockDim.x) {
    snap5[t] = snap_value((uint32_t)t, 0xF8u, 4u, 5u);
    snap6[t] = snap_value((uint32_t)t, 0xFCu, 2u, 6u);
  }
}

// Stages block (bx, by) into `t` with the 32 lanes of one warp and returns
// the block's sum of squared pixel values (all lanes).
__device__ __forceinline__ int stage_block(BlockTab &t, const uint8_t *__restrict__ rgb, int width, int bx, int by,
                                           int lane) {
  int sq = 0;
  uint32_t pk = 0;
  if (lane < 16) {
    const int r = lane >> 2, c = lane & 3;
    const uint8_t *p = rgb + ((size_t)(4 * by + r) * width + 4 * bx + c) * 3;
    const uint32_t R = p[0], G = p[1], B = p[2];
    const float third = __fdiv_rn(1.0f, 3.0f);
    const float fr = __uint2float_rn(R), fg = __uint2float_rn(G), fb = __uint2float_rn(B);
    const float qr = __fmul_rn(fr, third), qg = __fmul_rn(fg, third), qb = __fmul_rn(fb, third);
    const float4 P = make_float4(fr, fg, fb, 0.0f), Z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float4 Q = make_float4(qr, qg, qb, 0.0f);
    const float4 Q2 = make_float4(__fadd_rn(qr, qr), __fadd_rn(qg, qg), __fadd_rn(qb, qb), 0.0f);
    // (A, B) per index: 0: (px, 0), 1: (0, px), 2: (2q, q), 3: (q, 2q)
    const float4 va[4] = {P, Z, Q2, Q}, vb[4] = {Z, P, Q, Q2};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      t.ab[lane][0][k] = make_float2(va[k].x, va[k].y);
      t.ab[lane][1][k] = make_float2(va[k].z, vb[k].x);
      t.ab[lane][2][k] = make_float2(vb[k].y, vb[k].z);
    }
    pk = R | (G << 8) | (B << 16);
    sq = (int)(R * R + G * G + B * B);
  }
  // channel bytes of each group of four pixels
  const int c = lane >> 2, g = lane & 3;
  const uint32_t p0 = __shfl_sync(kFull, pk, 4 * g + 0), p1 = __shfl_sync(kFull, pk, 4 * g + 1);
  const uint32_t p2 = __shfl_sync(kFull, pk, 4 * g + 2), p3 = __shfl_sync(kFull, pk, 4 * g + 3);
  if (lane < 12) {
    const uint32_t sh = 8 * c;
    t.pg[c][g] = ((p0 >> sh) & 0xFF) | (((p1 >> sh) & 0xFF) << 8) | (((p2 >> sh) & 0xFF) << 16) |
                 (((p3 >> sh) & 0xFF) << 24);
  }
  __syncwarp();
  return __reduce_add_sync(kFull, sq);
}

// Weight sums of the refit for index word `cand`, accumulated in the
// reference's order (codec/dxt_image.cpp:307-312) from the per-index constants
// wk[index] = (a*a, b*b, a*b).
__device__ __forceinline__ WeightSums weight_sums(uint32_t cand, const float4 *wk) {
  float asq = 0.f, bsq = 0.f, ab = 0.f;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float4 w = wk[(cand >> (2 * i)) & 3u];
    asq = __fadd_rn(asq, w.x);
    bsq = __fadd_rn(bsq, w.y);
    ab = __fadd_rn(ab, w.z);
  }
  WeightSums r;
  r.asq = asq;
  r.bsq = bsq;
  r.ab = ab;
  r.f = __frcp_rn(__fsub_rn(__fmul_rn(asq, bsq), __fmul_rn(ab, ab)));
  return r;
}

// The per-index constants (a*a, b*b, a*b) with a, b as the reference computes
// them: a = (3-order)/3.0f, b = order/3.0f.
__device__ __forceinline__ void build_weight_table(float4 *wk) {
  if (threadIdx.x < 4) {
    const float order = threadIdx.x == 0 ? 0.f : threadIdx.x == 1 ? 3.f : threadIdx.x == 2 ? 1.f : 2.f;
    const float a = __fdiv_rn(__fsub_rn(3.0f, order), 3.0f), b = __fdiv_rn(order, 3.0f);
    wk[threadIdx.x] = make_float4(__fmul_rn(a, a), __fmul_rn(b, b), __fmul_rn(a, b), 0.0f);
  }
}

// Byte selector for __byte_perm from one byte of an index word: the four 2-bit
// indices of a group of pixels, spread to nibbles.
__device__ __forceinline__ uint32_t spread_nibbles(uint32_t b) {
  b = (b | (b << 4)) & 0x0F0Fu;
  return (b | (b << 2)) & 0x3333u;
}

// x86 cvttss2si of v followed by max(0, min(255, .)) (codec/dxt_image.cpp:330-331):
// NaN and |v| >= 2^31 convert to INT_MIN and therefore clamp to 0.
__device__ __forceinline__ uint32_t quantize_endpoint(float v) {
  float w = (v < 2147483648.0f) ? v : 0.0f;  // also maps NaN to 0
  w = fminf(fmaxf(w, 0.0f), 255.0f);
  return __float_as_uint(__fadd_rd(w, 8388608.0f)) - 0x4B000000u;  // floor(w)
}

__device__ __forceinline__ uint32_t pack565(uint32_t r, uint32_t g, uint32_t b) {
  return ((r & 0xF8u) << 8) | ((g & 0xFCu) << 3) | (b >> 3);
}

// Evaluates candidate `cand` on the staged block. Returns err_diff, or
// kInvalid when the refit would swap the endpoints (the candidate is skipped).
// `own` is the block's stb interp: AssignIndices with it is the identity
// (blk == blk2), which keeps the stb block with err_diff 0 and no refit.
// ws holds the candidate's weight sums.
__device__ __forceinline__ int eval_candidate(const BlockTab &t, const PixelGroups &pg, const uint8_t *snap5,
                                              const uint8_t *snap6, uint32_t cand, const WeightSums &ws,
                                              uint32_t own, int orig_err, int sumsq, uint32_t &eps, int &refit) {
  if (cand == own) {
    eps = 0;
    refit = 0;
    return 0;
  }
  refit = 1;
  // refit sums, pixel by pixel in the reference's order (codec/dxt_image.cpp:298-318)
  float ax0 = 0.f, ax1 = 0.f, ax2 = 0.f, bx0 = 0.f, bx1 = 0.f, bx2 = 0.f;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const uint32_t k = (cand >> (2 * i)) & 3u;
    const float2 u = t.ab[i][0][k], v = t.ab[i][1][k], w = t.ab[i][2][k];
    ax0 = __fadd_rn(ax0, u.x);
    bx0 = __fadd_rn(bx0, v.y);
    ax1 = __fadd_rn(ax1, u.y);
    bx1 = __fadd_rn(bx1, w.x);
    ax2 = __fadd_rn(ax2, v.x);
    bx2 = __fadd_rn(bx2, w.y);
  }
  // 2x2 solve (codec/dxt_image.cpp:320-326)
  const float f = ws.f, asq = ws.asq, bsq = ws.bsq, ab = ws.ab;
  const float p1r = __fmul_rn(f, __fsub_rn(__fmul_rn(ax0, bsq), __fmul_rn(bx0, ab)));
  const float p1g = __fmul_rn(f, __fsub_rn(__fmul_rn(ax1, bsq), __fmul_rn(bx1, ab)));
  const float p1b = __fmul_rn(f, __fsub_rn(__fmul_rn(ax2, bsq), __fmul_rn(bx2, ab)));
  const float p2r = __fmul_rn(f, __fsub_rn(__fmul_rn(bx0, asq), __fmul_rn(ax0, ab)));
  const float p2g = __fmul_rn(f, __fsub_rn(__fmul_rn(bx1, asq), __fmul_rn(ax1, ab)));
  const float p2b = __fmul_rn(f, __fsub_rn(__fmul_rn(bx2, asq), __fmul_rn(ax2, ab)));
  // quantise + snap (codec/dxt_image.cpp:329-341)
  const uint32_t e1r = snap5[quantize_endpoint(__fadd_rn(p1r, 0.5f))];
  const uint32_t e1g = snap6[quantize_endpoint(__fadd_rn(p1g, 0.5f))];
  const uint32_t e1b = snap5[quantize_endpoint(__fadd_rn(p1b, 0.5f))];
  const uint32_t e2r = snap5[quantize_endpoint(__fadd_rn(p2r, 0.5f))];
  const uint32_t e2g = snap6[quantize_endpoint(__fadd_rn(p2g, 0.5f))];
  const uint32_t e2b = snap5[quantize_endpoint(__fadd_rn(p2b, 0.5f))];
  const uint32_t q1 = pack565(e1r, e1g, e1b), q2 = pack565(e2r, e2g, e2b);
  if (q1 <= q2) return kInvalid;  // LogicalToPhysical would swap: skipped
  eps = q1 | (q2 << 16);
  // 4-colour palette of the refit (LerpChannels 1/3, 2/3, :346-347), one word
  // per channel holding the channel's four palette bytes
  const uint32_t wr = e1r | (e2r << 8) | (((2 * e1r + e2r) / 3) << 16) | (((e1r + 2 * e2r) / 3) << 24);
  const uint32_t wg = e1g | (e2g << 8) | (((2 * e1g + e2g) / 3) << 16) | (((e1g + 2 * e2g) / 3) << 24);
  const uint32_t wb = e1b | (e2b << 8) | (((2 * e1b + e2b) / 3) << 16) | (((e1b + 2 * e2b) / 3) << 24);
  // SSE = sum|s|^2 - 2 sum s.pal[idx] + sum |pal[idx]|^2 over four-pixel groups:
  // __byte_perm gathers the indexed palette bytes, dp4a multiplies-adds them.
  uint32_t cross = 0, norm = 0;
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const uint32_t sel = spread_nibbles((cand >> (8 * g)) & 0xFFu);
    const uint32_t vr = __byte_perm(wr, 0u, sel), vg = __byte_perm(wg, 0u, sel), vb = __byte_perm(wb, 0u, sel);
    cross = __dp4a(pg.w[0][g], vr, cross);
    cross = __dp4a(pg.w[1][g], vg, cross);
    cross = __dp4a(pg.w[2][g], vb, cross);
    norm = __dp4a(vr, vr, norm);
    norm = __dp4a(vg, vg, norm);
    norm = __dp4a(vb, vb, norm);
  }
  const int sse = sumsq - 2 * (int)cross + (int)norm;
  return (int)((uint32_t)sse / 48u) - orig_err;
}

// ---- the same evaluation from integer sums --------------------------------------
// The refit's inputs are small integers: with order o = {0, 3, 1, 2}[index] the
// sums are bx = S / 3 and ax = (3 T - S) / 3, S = sum px * o (four dp4a per
// channel) and T = sum px. The reference accumulates px * a and px * b in float,
// pixel by pixel; its rounding only matters where the refitted endpoint + 0.5
// falls next to an integer at which the snapped value changes. So the endpoints
// are computed from the exact sums and the candidate is decided where all six
// keep clear of such an integer by more than the two computations can differ; the
// others (ties in the small rational grid of the endpoints, mostly: about 1% of
// the candidates on the test streams) go through the reference's own float steps
// (refit_exact).
//
// Bound: with u = 2^-24, 16 terms of relative error <= 2u (px * fl(1/3)) added in
// 15 roundings give ax, bx to 17.1u; here each sum is one product (2u). The two
// products, their difference and the products with the weight sums' float values
// (the same in both) add 4u of ax * bsq + bx * ab, which is at most
// T * max(asq, bsq): |difference| <= 23.1u * |f| * T * max(asq, bsq) + 5u * |p| plus
// the two roundings of p + 0.5 (each <= 2^-17). |p| <= 260 covers every value that
// the clamp to [0, 255] leaves. Where that is not below a quarter (a degenerate
// word, all indices equal: f huge, infinite or NaN), refit_exact decides.
constexpr float kRefitRel = 1.46e-6f;  // > 23.1u (1.05 x)
constexpr float kRefitAbs = 1.0e-4f;   // > 260 * 5u + 2^-16

// The pixels of N blocks: [0 .. 2][block] the channel's bytes of pixels 4g .. 4g+3 in
// word g, [3][block] the channels' sums, then the sum of squares over all. A
// vector of adjacent blocks is contiguous, so lanes that work on different blocks
// read it without bank conflicts (a block by itself, 64 bytes, put every other
// block into the same banks: 11 million conflicts a 1080p frame).
template <int N>
struct __align__(16) PixBlocks {
  uint32_t w[4][N][4];
};
// Block k of them.
template <int N>
struct PixBlock {
  const PixBlocks<N> &t;
  int k;
  __device__ __forceinline__ uint4 vec(int c) const { return *reinterpret_cast<const uint4 *>(t.w[c][k]); }
  __device__ __forceinline__ uint32_t word(int c, int g) const { return t.w[c][k][g]; }
};

// The snap tables with, per value, whether the snapped value differs from that
// of the value before (bit 31); the snapped value in the low byte.
constexpr uint32_t kSnapLow = 0x80000000u;
struct SnapTables {
  uint32_t five[256], six[256];
};
__device__ __forceinline__ void build_snap_edges(SnapTables &t) {
  for (int i = threadIdx.x; i < 512; i += blockDim.x) {
    const uint32_t x = (uint32_t)i & 255u, keep = i < 256 ? 0xF8u : 0xFCu, step = i < 256 ? 4u : 2u, sh = i < 256 ? 5u : 6u;
    const uint32_t v = snap_value(x, keep, step, sh), lo = x > 0u ? snap_value(x - 1u, keep, step, sh) : v;
    (i < 256 ? t.five : t.six)[x] = v | (lo != v ? kSnapLow : 0u);
  }
}

// The channel words (bytes of pixels 0 .. 3) of pixel row y of block column bx:
// three aligned words of the frame (rows and blocks are a multiple of 4 bytes
// apart).
__device__ __forceinline__ void load_channels(const uint8_t *__restrict__ rgb, int width, int bx, int y, uint32_t &c0,
                                              uint32_t &c1, uint32_t &c2) {
  const uint32_t *p = reinterpret_cast<const uint32_t *>(rgb + ((size_t)y * width + 4 * bx) * 3);
  const uint32_t w0 = __ldg(p), w1 = __ldg(p + 1), w2 = __ldg(p + 2);  // R0G0B0R1 G1B1R2G2 B2R3G3B3
  c0 = __byte_perm(__byte_perm(w0, w1, 0x0630), w2, 0x5210);
  c1 = __byte_perm(__byte_perm(w0, w1, 0x0741), w2, 0x6210);
  c2 = __byte_perm(__byte_perm(w0, w1, 0x0052), w2, 0x7410);
}

// A refit's six endpoint values as entries of the snap tables: ep1's r, g, b, then
// ep2's.
struct RefitValues {
  uint32_t snap[6];
};

// From the exact sums; false where the float steps may give another value.
template <int N>
__device__ __forceinline__ bool refit_quick(const PixBlock<N> t, const SnapTables &st, uint32_t cand,
                                            const WeightSums &ws, RefitValues &r) {
  const float third = __fdiv_rn(1.0f, 3.0f);
  uint32_t ord[4];
#pragma unroll
  for (int g = 0; g < 4; ++g) ord[g] = __byte_perm(0x02010300u, 0u, spread_nibbles((cand >> (8 * g)) & 0xFFu));
  const uint4 sums = t.vec(3);
  const uint32_t sum[3] = {sums.x, sums.y, sums.z};
  const float tmax = __uint2float_rn(max(sum[0], max(sum[1], sum[2])));
  const float margin =
      __fmaf_rn(__fmul_rn(__fmul_rn(kRefitRel, tmax), fabsf(ws.f)), fmaxf(ws.asq, ws.bsq), kRefitAbs);
  // Values as w + 2048, whose last 12 bits are w's fraction (rounded by half a unit,
  // which `near`, the margin in units, covers: one unit for its own rounding down,
  // one for this). With k = floor(w + margin), a fraction of w + margin of at
  // least twice the margin puts the reference's value at k as well; below that it is k
  // or k - 1, which is no matter where both snap to the same value.
  const uint32_t near = (uint32_t)__float2int_rz(__fmul_rn(margin, 4096.0f)) + 2u, span = 2u * near;
  uint32_t edge = 0;  // bit 31: a value that may be k or k - 1 where they snap differently
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const uint4 pg = t.vec(c);
    const uint32_t S = __dp4a(pg.w, ord[3], __dp4a(pg.z, ord[2], __dp4a(pg.y, ord[1], __dp4a(pg.x, ord[0], 0u))));
    const float b = __fmul_rn(__uint2float_rn(S), third), a = __fmul_rn(__uint2float_rn(3u * sum[c] - S), third);
    const float v1 = __fmaf_rn(ws.f, __fsub_rn(__fmul_rn(a, ws.bsq), __fmul_rn(b, ws.ab)), 0.5f);
    const float v2 = __fmaf_rn(ws.f, __fsub_rn(__fmul_rn(b, ws.asq), __fmul_rn(a, ws.ab)), 0.5f);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float w = fminf(fmaxf(h ? v2 : v1, 0.5f), 255.5f);
      const uint32_t x = __float_as_uint(__fadd_rn(w, 2048.0f)) + near;
      const uint32_t e = (c == 1 ? st.six : st.five)[(x >> 12) & 0xFFu];
      edge |= ((x & 0xFFFu) - span) & e;
      r.snap[3 * h + c] = e;
    }
  }
  return (int)edge >= 0 && margin < 0.25f;  // false for a NaN or infinite margin
}

// By the reference's own steps (codec/dxt_image.cpp:298-331).
template <int N>
__device__ __forceinline__ void refit_exact(const PixBlock<N> t, const SnapTables &st, uint32_t cand,
                                            const WeightSums &ws, RefitValues &r) {
  const float third = __fdiv_rn(1.0f, 3.0f), third2 = __fadd_rn(third, third);
  float ax[3] = {0.f, 0.f, 0.f}, bx[3] = {0.f, 0.f, 0.f};
#pragma unroll 1
  for (int g = 0; g < 4; ++g) {
    const uint32_t w[3] = {t.word(0, g), t.word(1, g), t.word(2, g)}, idx = cand >> (8 * g);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t k = (idx >> (2 * i)) & 3u;
      // px * a, px * b of the index: (1, 0), (0, 1), (2/3, 1/3), (1/3, 2/3)
      const float lo = (k & 2u) ? third2 : 1.0f, hi = (k & 2u) ? third : 0.0f;
      const float fa = (k & 1u) ? hi : lo, fb = (k & 1u) ? lo : hi;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float px = __uint2float_rn((w[c] >> (8 * i)) & 0xFFu);
        ax[c] = __fadd_rn(ax[c], __fmul_rn(px, fa));
        bx[c] = __fadd_rn(bx[c], __fmul_rn(px, fb));
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float p1 = __fmul_rn(ws.f, __fsub_rn(__fmul_rn(ax[c], ws.bsq), __fmul_rn(bx[c], ws.ab)));
    const float p2 = __fmul_rn(ws.f, __fsub_rn(__fmul_rn(bx[c], ws.asq), __fmul_rn(ax[c], ws.ab)));
    const uint32_t *s = c == 1 ? st.six : st.five;
    r.snap[c] = s[quantize_endpoint(__fadd_rn(p1, 0.5f))];
    r.snap[3 + c] = s[quantize_endpoint(__fadd_rn(p2, 0.5f))];
  }
}

// One channel of it: the pixels' bytes, the channel's snap table; entries of ep1's and
// ep2's value.
__device__ __forceinline__ void refit_exact_channel(uint4 pg, const uint32_t *snap, uint32_t cand,
                                                    const WeightSums &ws, uint32_t &snap1, uint32_t &snap2) {
  const float third = __fdiv_rn(1.0f, 3.0f), third2 = __fadd_rn(third, third);
  float ax = 0.f, bx = 0.f;
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const uint32_t w = g == 0 ? pg.x : g == 1 ? pg.y : g == 2 ? pg.z : pg.w, idx = cand >> (8 * g);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t k = (idx >> (2 * i)) & 3u;
      const float lo = (k & 2u) ? third2 : 1.0f, hi = (k & 2u) ? third : 0.0f;
      const float fa = (k & 1u) ? hi : lo, fb = (k & 1u) ? lo : hi;
      const float px = __uint2float_rn((w >> (8 * i)) & 0xFFu);
      ax = __fadd_rn(ax, __fmul_rn(px, fa));
      bx = __fadd_rn(bx, __fmul_rn(px, fb));
    }
  }
  const float p1 = __fmul_rn(ws.f, __fsub_rn(__fmul_rn(ax, ws.bsq), __fmul_rn(bx, ws.ab)));
  const float p2 = __fmul_rn(ws.f, __fsub_rn(__fmul_rn(bx, ws.asq), __fmul_rn(ax, ws.ab)));
  snap1 = snap[quantize_endpoint(__fadd_rn(p1, 0.5f))];
  snap2 = snap[quantize_endpoint(__fadd_rn(p2, 0.5f))];
}

// err_diff of the refitted candidate (kInvalid where its endpoints would swap)
// and its packed endpoints.
template <int N>
__device__ __forceinline__ int refit_error(const PixBlock<N> t, const RefitValues &r, uint32_t cand, int orig_err,
                                           uint32_t &eps) {
  const uint32_t q1 = ((r.snap[0] << 8) & 0xF800u) | ((r.snap[1] << 3) & 0x07E0u) | ((r.snap[2] >> 3) & 0x1Fu);
  const uint32_t q2 = ((r.snap[3] << 8) & 0xF800u) | ((r.snap[4] << 3) & 0x07E0u) | ((r.snap[5] >> 3) & 0x1Fu);
  eps = q1 | (q2 << 16);
  // the channel's four palette bytes: e1, e2, (2 e1 + e2) / 3, (e1 + 2 e2) / 3; x / 3
  // is (x * 683) >> 11 for x <= 765, here shifted into its byte
  uint32_t pal[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const uint32_t ends = __byte_perm(r.snap[c], r.snap[3 + c], 0x0040) & 0xFFFFu;
    const uint32_t x2 = __dp4a(ends, 0x0102u, 0u), x3 = __dp4a(ends, 0x0201u, 0u);
    pal[c] = ends | ((x2 * (683u << 5)) & 0x00FF0000u) | ((x3 * (683u << 13)) & 0xFF000000u);
  }
  uint32_t cross = 0, norm = 0;
  const uint4 pg[3] = {t.vec(0), t.vec(1), t.vec(2)};
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const uint32_t sel = spread_nibbles((cand >> (8 * g)) & 0xFFu);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const uint32_t v = __byte_perm(pal[c], 0u, sel);
      cross = __dp4a(g == 0 ? pg[c].x : g == 1 ? pg[c].y : g == 2 ? pg[c].z : pg[c].w, v, cross);
      norm = __dp4a(v, v, norm);
    }
  }
  const int sse = (int)t.word(3, 3) - 2 * (int)cross + (int)norm;
  return q1 > q2 ? (int)((uint32_t)sse / 48u) - orig_err : kInvalid;
}

// refit_exact and refit_error of up to kByChannels candidates by a warp, a lane per
// channel: few candidates need the float steps, and a pass with a lane per
// candidate costs as much for one as for 32 (560 instructions against 330). get(q):
// candidate q of n; returns candidate `lane`'s err_diff and endpoints. All lanes call.
constexpr int kByChannels = 10;
template <int N>
struct ExactCase {
  PixBlock<N> px;
  uint32_t cand;
  float4 d;  // its weight sums
  int orig;
};
template <class Get>
__device__ __forceinline__ uint2 refit_by_channels(const SnapTables &st, int n, int lane, Get get) {
  const int q = lane / 3, c = lane - 3 * q;
  uint32_t v1 = 0, v2 = 0;
  if (q < n) {
    const auto x = get(q);
    refit_exact_channel(x.px.vec(c), c == 1 ? st.six : st.five, x.cand, WeightSums{x.d.x, x.d.y, x.d.z, x.d.w}, v1, v2);
  }
  RefitValues r;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    r.snap[k] = __shfl_sync(kFull, v1, 3 * lane + k);
    r.snap[3 + k] = __shfl_sync(kFull, v2, 3 * lane + k);
  }
  uint32_t eps = 0;
  int e = kInvalid;
  if (lane < n) {
    const auto x = get(lane);
    e = refit_error(x.px, r, x.cand, x.orig, eps);
  }
  return make_uint2((uint32_t)e, eps);
}

}  // namespace mptc
