// Endpoint images and stream decode on the GPU.
//
// Encoder side: the two endpoint images of a frame (ep1, ep2 of every final
// block, RGB565) go to YCoCg-667 (codec/image_processing.cpp:10-27), then each
// 64x64 tile of each plane gets the 6-level integer 5/3 lifting wavelet
// (codec/image_processing.h:292-330, codec/wavelet.cpp:30-127): per level
// dim = 64, 32, ..., 2 a column pass then a row pass over the top-left
// dim x dim corner. Coefficients are wrapped to int8 and offset by 128
// (codec/image_utils.h:218-237, pixel_traits.h:261-273).
//
// Decoder side: the inverse (codec/decoder.cpp:68-107, wavelet.cpp:69-155;
// dim = 2, ..., 64, rows then columns), YCoCg-667 -> RGB565 in int8
// arithmetic (decoder.cpp:24-41, 109-201), and the index words from the motion
// codes (decoder.cpp:203-254): unique blocks take the next palette entry in
// raster order, inter blocks copy from the previous frame, intra blocks copy
// from an earlier block of the same frame. The intra copies form chains that
// every block follows by itself, shortening them for the others on the way,
// instead of the reference's raster loop.
//
// Both transforms: one CTA per (64x64 tile, plane), two int16 tiles in shared
// memory (source and destination of each lifting pass).
#pragma once

#include <cstdint>

#include "lookback.cuh"

namespace mptc {

constexpr int kTile = 64;                 // endpoint tile edge (blocks)
constexpr int kTileElems = kTile * kTile;
constexpr int kCodecThreads = 256;

// The lifting passes. What bounds them is latency: a tile is 12 dependent
// passes (two per level) and a frame has few tiles (240 planes at 2048x1280, at
// most two per SM), so a pass has to be short: each thread takes a piece of
// K outputs of each half of a line into registers and computes its
// halo's details itself, one barrier a pass; the levels up to 16x16 are one
// warp's work and need none. Rows of 66 elements (33 words) keep both
// directions free of bank conflicts: a row pass has its lanes in a column, a
// column pass takes two adjacent columns per lane as one word.
// One thread per output, two steps and barriers a pass, took 31 us for a
// 2048x1280 frame forward and 52 inverse; now 7.6 us forward, and 11.5 inverse
// together with the motion codes.
constexpr int kPitch = kTile + 2;
struct __align__(16) LiftTile {
  uint32_t w[kTile * kPitch / 2];
};

__device__ __forceinline__ int lo16(uint32_t w) { return (int)(int16_t)(w & 0xFFFFu); }
__device__ __forceinline__ int hi16(uint32_t w) { return (int)(int16_t)(w >> 16); }
__device__ __forceinline__ uint32_t pack16(int lo, int hi) { return ((uint32_t)lo & 0xFFFFu) | ((uint32_t)hi << 16); }

// A piece of a forward line (codec/wavelet.cpp:30-66): e[2 + i] = element i of
// the piece, i = -2 .. 2K (the halo unread where the line ends); details
// hi[k] = e[2k+1] - (e[2k] + e[2k+2]) / 2, approximations lo[k] = e[2k] +
// (hi[k-1] + hi[k] + 2) / 4, mirrored at both ends, each stored in 16 bits.
template <int K>
__device__ __forceinline__ void forward_piece(int (&e)[2 * K + 3], bool first, bool last, int (&lo)[K], int (&hi)[K]) {
  if (last) e[2 * K + 2] = e[2 * K];
#pragma unroll
  for (int k = 0; k < K; ++k) hi[k] = (int)(int16_t)(e[2 * k + 3] - (e[2 * k + 2] + e[2 * k + 4]) / 2);
  int before = first ? hi[0] : (int)(int16_t)(e[1] - (e[0] + e[2]) / 2);
#pragma unroll
  for (int k = 0; k < K; ++k) {
    lo[k] = (int)(int16_t)(e[2 * k + 2] + (before + hi[k] + 2) / 4);
    before = hi[k];
  }
}

// Its inverse (codec/wavelet.cpp:69-99): s[k] = approximation k of the piece (k
// = 0 .. K), d[1 + k] = detail k (k = -1 .. K); even and odd elements.
template <int K>
__device__ __forceinline__ void inverse_piece(int (&s)[K + 1], int (&d)[K + 2], bool first, bool last, int (&even)[K],
                                              int (&odd)[K]) {
  if (first) d[0] = d[1];
#pragma unroll
  for (int k = 0; k < K; ++k) even[k] = (int)(int16_t)(s[k] - (d[k] + d[k + 1] + 2) / 4);
  const int after = last ? even[K - 1] : (int)(int16_t)(s[K] - (d[K] + d[K + 1] + 2) / 4);
#pragma unroll
  for (int k = 0; k < K; ++k) odd[k] = (int)(int16_t)(d[k + 1] + (even[k] + (k + 1 < K ? even[k + 1] : after)) / 2);
}

// One pass over the top-left DIM x DIM corner, src -> dst, by `threads` threads.
template <int DIM, int K>
__device__ __forceinline__ void forward_rows(const LiftTile &src, LiftTile &dst, int tid, int threads) {
  constexpr int kHalf = DIM / 2, kPieces = kHalf / K;
  int16_t *out = reinterpret_cast<int16_t *>(dst.w);
  for (int t = tid; t < DIM * kPieces; t += threads) {
    const int row = t % DIM, k0 = t / DIM * K;
    const uint32_t *in = src.w + row * (kPitch / 2);
    int e[2 * K + 3], lo[K], hi[K];
    const uint32_t left = in[max(k0 - 1, 0)];
    e[0] = lo16(left), e[1] = hi16(left);
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const uint32_t w = in[k0 + k];
      e[2 * k + 2] = lo16(w), e[2 * k + 3] = hi16(w);
    }
    e[2 * K + 2] = lo16(in[min(k0 + K, kHalf - 1)]);
    forward_piece<K>(e, k0 == 0, k0 + K == kHalf, lo, hi);
#pragma unroll
    for (int k = 0; k < K; ++k) {
      out[row * kPitch + k0 + k] = (int16_t)lo[k];
      out[row * kPitch + kHalf + k0 + k] = (int16_t)hi[k];
    }
  }
}

template <int DIM, int K>
__device__ __forceinline__ void forward_columns(const LiftTile &src, LiftTile &dst, int tid, int threads) {
  constexpr int kHalf = DIM / 2, kPieces = kHalf / K, kRow = kPitch / 2;
  for (int t = tid; t < kHalf * kPieces; t += threads) {  // kHalf column pairs
    const int c = t % kHalf, k0 = t / kHalf * K;
    const uint32_t *in = src.w + c;
    int e[2 * K + 3], f[2 * K + 3], lo[K], hi[K], lo2[K], hi2[K];
#pragma unroll
    for (int i = 0; i < 2 * K + 3; ++i) {
      const uint32_t w = in[min(max(2 * k0 - 2 + i, 0), DIM - 1) * kRow];
      e[i] = lo16(w), f[i] = hi16(w);
    }
    forward_piece<K>(e, k0 == 0, k0 + K == kHalf, lo, hi);
    forward_piece<K>(f, k0 == 0, k0 + K == kHalf, lo2, hi2);
#pragma unroll
    for (int k = 0; k < K; ++k) {
      dst.w[(k0 + k) * kRow + c] = pack16(lo[k], lo2[k]);
      dst.w[(kHalf + k0 + k) * kRow + c] = pack16(hi[k], hi2[k]);
    }
  }
}

template <int DIM, int K>
__device__ __forceinline__ void inverse_rows(const LiftTile &src, LiftTile &dst, int tid, int threads) {
  constexpr int kHalf = DIM / 2, kPieces = kHalf / K;
  const int16_t *in = reinterpret_cast<const int16_t *>(src.w);
  for (int t = tid; t < DIM * kPieces; t += threads) {
    const int row = t % DIM, k0 = t / DIM * K;
    const int16_t *a = in + row * kPitch;
    int s[K + 1], d[K + 2], even[K], odd[K];
#pragma unroll
    for (int k = 0; k <= K; ++k) s[k] = a[min(k0 + k, kHalf - 1)];
#pragma unroll
    for (int k = 0; k < K + 2; ++k) d[k] = a[kHalf + min(max(k0 - 1 + k, 0), kHalf - 1)];
    inverse_piece<K>(s, d, k0 == 0, k0 + K == kHalf, even, odd);
#pragma unroll
    for (int k = 0; k < K; ++k) dst.w[row * (kPitch / 2) + k0 + k] = pack16(even[k], odd[k]);
  }
}

template <int DIM, int K>
__device__ __forceinline__ void inverse_columns(const LiftTile &src, LiftTile &dst, int tid, int threads) {
  constexpr int kHalf = DIM / 2, kPieces = kHalf / K, kRow = kPitch / 2;
  for (int t = tid; t < kHalf * kPieces; t += threads) {
    const int c = t % kHalf, k0 = t / kHalf * K;
    const uint32_t *in = src.w + c;
    int s[K + 1], d[K + 2], even[K], odd[K], s2[K + 1], d2[K + 2], even2[K], odd2[K];
#pragma unroll
    for (int k = 0; k <= K; ++k) {
      const uint32_t w = in[min(k0 + k, kHalf - 1) * kRow];
      s[k] = lo16(w), s2[k] = hi16(w);
    }
#pragma unroll
    for (int k = 0; k < K + 2; ++k) {
      const uint32_t w = in[(kHalf + min(max(k0 - 1 + k, 0), kHalf - 1)) * kRow];
      d[k] = lo16(w), d2[k] = hi16(w);
    }
    inverse_piece<K>(s, d, k0 == 0, k0 + K == kHalf, even, odd);
    inverse_piece<K>(s2, d2, k0 == 0, k0 + K == kHalf, even2, odd2);
#pragma unroll
    for (int k = 0; k < K; ++k) {
      dst.w[(2 * (k0 + k)) * kRow + c] = pack16(even[k], even2[k]);
      dst.w[(2 * (k0 + k) + 1) * kRow + c] = pack16(odd[k], odd2[k]);
    }
  }
}

// grid (bw/64, bh/64, 6 planes: Y, Co, Cg of endpoint 1, then of endpoint 2),
// one plane of one tile per CTA. coeff: 6 planes of bw*bh bytes,
// [Y1 | Co1 | Cg1 | Y2 | Co2 | Cg2], each plane raster order over the image;
// written in words where it is aligned to them (bw is a multiple of 64).
__global__ void __launch_bounds__(kCodecThreads) endpoint_forward_kernel(const uint64_t *__restrict__ blocks, int bw,
                                                                         int bh, uint8_t *__restrict__ coeff) {
  __shared__ LiftTile a, b;
  depend();
  release_next();
  const int tid = threadIdx.x, tx = blockIdx.x * kTile, ty = blockIdx.y * kTile, plane = blockIdx.z;
  const int ep = plane / 3, channel = plane - 3 * ep;
  const size_t n = (size_t)bw * bh;
  const uint32_t *src = reinterpret_cast<const uint32_t *>(blocks + (size_t)ty * bw + tx);
  int16_t *a16 = reinterpret_cast<int16_t *>(a.w);
#pragma unroll
  for (int r = 0; r < kTileElems / kCodecThreads; ++r) {
    const int e = r * kCodecThreads + tid, y = e >> 6, x = e & 63;
    const uint32_t lo = src[2 * ((size_t)y * bw + x)];
    const int c = (int)(ep ? (lo >> 16) : (lo & 0xFFFFu));
    const int r5 = c >> 11, g6 = (c >> 5) & 63, b5 = c & 31;
    const int co = r5 - b5, t = r5 + b5 + (b5 >> 4), cg = g6 - t;
    a16[y * kPitch + x] = (int16_t)(channel == 0 ? t + cg / 2 : (channel == 1 ? co : cg));
  }
  __syncthreads();
  forward_columns<64, 4>(a, b, tid, kCodecThreads);
  __syncthreads();
  forward_rows<64, 8>(b, a, tid, kCodecThreads);
  __syncthreads();
  forward_columns<32, 2>(a, b, tid, kCodecThreads);
  __syncthreads();
  forward_rows<32, 2>(b, a, tid, kCodecThreads);
  __syncthreads();
  if (tid < 32) {
    forward_columns<16, 2>(a, b, tid, 32);
    __syncwarp();
    forward_rows<16, 4>(b, a, tid, 32);
    __syncwarp();
    forward_columns<8, 1>(a, b, tid, 32);
    __syncwarp();
    forward_rows<8, 1>(b, a, tid, 32);
    __syncwarp();
    forward_columns<4, 1>(a, b, tid, 32);
    __syncwarp();
    forward_rows<4, 1>(b, a, tid, 32);
    __syncwarp();
    forward_columns<2, 1>(a, b, tid, 32);
    __syncwarp();
    forward_rows<2, 1>(b, a, tid, 32);
  }
  __syncthreads();
  uint8_t *out = coeff + (size_t)plane * n + (size_t)ty * bw + tx;
  const bool words = (reinterpret_cast<uintptr_t>(coeff) & 3u) == 0;
#pragma unroll
  for (int r = 0; r < kTileElems / 4 / kCodecThreads; ++r) {
    const int e = r * kCodecThreads + tid, y = e >> 4, x = 4 * (e & 15);
    const uint32_t w0 = a.w[(y * kPitch + x) / 2], w1 = a.w[(y * kPitch + x) / 2 + 1];
    // the coefficients wrap to int8 and are offset by 128
    const uint32_t v = __byte_perm(w0, w1, 0x6420) ^ 0x80808080u;
    uint8_t *o = out + (size_t)y * bw + x;
    if (words) {
      *reinterpret_cast<uint32_t *>(o) = v;
    } else {
      o[0] = (uint8_t)v, o[1] = (uint8_t)(v >> 8), o[2] = (uint8_t)(v >> 16), o[3] = (uint8_t)(v >> 24);
    }
  }
}

// One plane of one tile: coefficients -> the plane's values in int8 (planes:
// as coeff), by one CTA. Where coeff is aligned to words it is read in words.
__device__ __forceinline__ void inverse_tile(const uint8_t *__restrict__ coeff, int bw, size_t off, LiftTile &a,
                                             LiftTile &b, uint8_t *__restrict__ planes) {
  const int tid = threadIdx.x;
  const bool words = (reinterpret_cast<uintptr_t>(coeff) & 3u) == 0;
#pragma unroll
  for (int r = 0; r < kTileElems / 4 / kCodecThreads; ++r) {
    const int e = r * kCodecThreads + tid, y = e >> 4, x = 4 * (e & 15);
    const uint8_t *i = coeff + off + (size_t)y * bw + x;
    uint32_t v;
    if (words)
      v = *reinterpret_cast<const uint32_t *>(i);
    else
      v = i[0] | (uint32_t)i[1] << 8 | (uint32_t)i[2] << 16 | (uint32_t)i[3] << 24;
    uint32_t *o = a.w + (y * kPitch + x) / 2;
    o[0] = pack16((int)(v & 255u) - 128, (int)(v >> 8 & 255u) - 128);
    o[1] = pack16((int)(v >> 16 & 255u) - 128, (int)(v >> 24) - 128);
  }
  __syncthreads();
  if (tid < 32) {
    inverse_rows<2, 1>(a, b, tid, 32);
    __syncwarp();
    inverse_columns<2, 1>(b, a, tid, 32);
    __syncwarp();
    inverse_rows<4, 1>(a, b, tid, 32);
    __syncwarp();
    inverse_columns<4, 1>(b, a, tid, 32);
    __syncwarp();
    inverse_rows<8, 1>(a, b, tid, 32);
    __syncwarp();
    inverse_columns<8, 1>(b, a, tid, 32);
    __syncwarp();
    inverse_rows<16, 4>(a, b, tid, 32);
    __syncwarp();
    inverse_columns<16, 2>(b, a, tid, 32);
  }
  __syncthreads();
  inverse_rows<32, 2>(a, b, tid, kCodecThreads);
  __syncthreads();
  inverse_columns<32, 2>(b, a, tid, kCodecThreads);
  __syncthreads();
  inverse_rows<64, 8>(a, b, tid, kCodecThreads);
  __syncthreads();
  inverse_columns<64, 4>(b, a, tid, kCodecThreads);
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kTileElems / 4 / kCodecThreads; ++r) {
    const int e = r * kCodecThreads + tid, y = e >> 4, x = 4 * (e & 15);
    const uint32_t *i = a.w + (y * kPitch + x) / 2;
    *reinterpret_cast<uint32_t *>(planes + off + (size_t)y * bw + x) = __byte_perm(i[0], i[1], 0x6420);
  }
}

// One endpoint word from its plane values, in the int8 arithmetic in which the
// reference stores them (decoder.cpp:24-41, 145-160).
__device__ __forceinline__ uint16_t endpoint_word(uint8_t y, uint8_t o, uint8_t c) {
  const int8_t Y = (int8_t)y, Co = (int8_t)o, Cg = (int8_t)c;
  const int8_t t = (int8_t)(Y - Cg / 2);
  const int8_t g = (int8_t)(Cg + t);
  const int8_t bb = (int8_t)((t - Co) / 2);
  const int8_t r = (int8_t)(bb + Co);
  uint16_t w = (uint16_t)(int16_t)r;
  w = (uint16_t)(w << 6);
  w |= (uint16_t)(int16_t)g;
  w = (uint16_t)(w << 5);
  w |= (uint16_t)(int16_t)bb;
  return w;
}

// --- index words from motion codes ---

constexpr uint32_t kDecBadRef = 1u, kDecBadUnique = 2u;

// A block's link: kLinkWord | its index word, or the earlier block that it copies.
constexpr uint64_t kLinkWord = 1ull << 32;

// First kernel of a frame. The first ntiles CTAs read the motion codes of
// kScanTile blocks each (tiles taken in order from *claim): a unique block takes
// palette[its rank among the unique blocks in raster order] (one-pass compaction,
// lookback.cuh), an inter block the previous frame's word, an intra block a link. The
// other CTAs are the inverse transform of the frame's tiles, which runs beside
// them. 11.5 us at 2048x1280; as three kernels, one after
// another, 52, 5 and 11 us.
__global__ void __launch_bounds__(kCodecThreads) decode_parts_kernel(
    const uint8_t *__restrict__ coeff, int bw, int bh, uint8_t *__restrict__ planes,
    const uint8_t *__restrict__ motion, const uint64_t *prev, int sa, const uint32_t *__restrict__ palette,
    uint32_t n_unique, int ntiles, uint64_t *state, uint32_t *claim, uint64_t *__restrict__ link,
    uint32_t *__restrict__ err, uint32_t *__restrict__ status) {
  __shared__ LiftTile a, b;
  __shared__ int s_tile;
  __shared__ uint32_t s_warp[8], s_before;
  depend();
  release_next();
  const int nblk = bw * bh, tid = threadIdx.x;
  if ((int)blockIdx.x >= ntiles) {
    const int tiles_x = bw / kTile, tiles = tiles_x * (bh / kTile);
    const int u = blockIdx.x - ntiles, plane = u / tiles, tile = u - plane * tiles;
    const int ty = tile / tiles_x, tx = tile - ty * tiles_x;
    inverse_tile(coeff, bw, (size_t)plane * nblk + (size_t)ty * kTile * bw + tx * kTile, a, b, planes);
    return;
  }
  if (tid == 0) s_tile = (int)atomicAdd(claim, 1u);
  __syncthreads();
  const int tile = s_tile, i0 = tile * kScanTile + 4 * tid;
  if ((unsigned)tile >= (unsigned)ntiles) {  // two frames of a decoder at the same time, for instance
    if (tid == 0) atomicOr(status, kDevBadScan);
    return;
  }
  unsigned uq = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = i0 + q;
    if (i >= nblk) break;
    const int x = motion[2 * i], y = motion[2 * i + 1];
    const int by = i / bw, bx = i - by * bw;
    if (x == 255 && y == 255) {
      uq |= 1u << q;
    } else if ((x & 0x80) && (y & 0x80)) {
      // linear index as the reference computes it (decoder.cpp:224-236)
      const long ref = (long)(by + (y & 0x7F) - sa) * bw + bx + (x & 0x7F) - sa;
      uint32_t v = 0;
      if (prev && ref >= 0 && ref < nblk) v = (uint32_t)(prev[ref] >> 32);
      else atomicOr(err, kDecBadRef);
      link[i] = kLinkWord | v;
    } else {
      const long ref = (long)(by + y - 2 * sa + 1) * bw + bx + x - sa;
      if (ref >= 0 && ref < i) {
        link[i] = (uint64_t)ref;
      } else {
        atomicOr(err, kDecBadRef);
        link[i] = kLinkWord;
      }
    }
  }
  uint32_t total;
  uint32_t off = cta_exclusive_scan(__popc(uq), s_warp, total);
  if (tid < 32) {
    const uint32_t before = lookback(state, tile, total, status);
    if (tid == 0) s_before = before;
  }
  __syncthreads();
  off += s_before;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if ((uq >> q) & 1u) {
      link[i0 + q] = kLinkWord | (off < n_unique ? palette[off] : 0u);
      ++off;
    }
  if (tile == ntiles - 1 && tid == 0 && s_before + total != n_unique) atomicOr(err, kDecBadUnique);
}

// Second kernel: each block follows its link to a word and writes its DXT1
// block. A link leads to an earlier block (or is the word that the decoder was made
// with), so the walk ends; on the way a block
// replaces its own link (which only it writes) by the one it has just read, so
// that the blocks behind it skip that part: with all of them walking at once a chain halves
// at each step, as in pointer jumping, but without a launch and a pass over
// memory per step (19 launches of 3.7 us before; 3.5 to 9 us now, by the chains). The scan's state is left
// zeroed for the next frame.
__global__ void __launch_bounds__(256) decode_link_kernel(const uint8_t *__restrict__ planes, int nblk, uint64_t *link,
                                                          uint64_t *__restrict__ state, int ntiles,
                                                          uint32_t *__restrict__ claim, uint64_t *__restrict__ out) {
  depend();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < ntiles) state[i] = 0ull;
  if (i == 0) *claim = 0u;
  if (i >= nblk) return;
  uint64_t w = ld_relaxed(link + i);
  uint8_t v[6];
#pragma unroll
  for (int p = 0; p < 6; ++p) v[p] = planes[(size_t)p * nblk + i];
  while (w < kLinkWord) {
    w = ld_relaxed(link + w);
    st_relaxed(link + i, w);
  }
  out[i] = (uint64_t)endpoint_word(v[0], v[1], v[2]) | ((uint64_t)endpoint_word(v[3], v[4], v[5]) << 16) | (w << 32);
}

}  // namespace mptc
