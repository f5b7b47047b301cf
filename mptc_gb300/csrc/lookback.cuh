// Ordered compactions in one pass: tile states and the look-back over them.
#pragma once
#include <cstdint>

#include "completion.cuh"

namespace mptc {

// ------------------------------------------------------ ordered compaction --
// Single-pass ordered compactions (decoupled look-back, Merrill & Garland,
// "Single-pass Parallel Prefix Scan with Decoupled Look-back", 2016): a CTA
// per tile of kScanTile blocks takes tiles in order from a zeroed counter,
// counts its tile, publishes the count, adds up its predecessors' published
// counts (or the first inclusive prefix among them) and scatters its items
// at the resulting offset. Tile states are 64-bit words, zeroed per frame:
// 0 = not yet published, kTileAgg | v = the tile's count v, kTilePre | v =
// the count of the tile and all tiles before it. A tile reads only tiles
// taken before it by running CTAs, so the look-back always ends; each wait
// is bounded like wait_done.
constexpr int kScanTile = 1024;  // blocks per tile: 256 threads x 4
constexpr uint64_t kTileAgg = 1ull << 62, kTilePre = 2ull << 62;

// Warp 0 of the CTA owning `tile`: publishes `count` and returns (in every
// lane) the sum of the counts of the tiles before it.
__device__ __forceinline__ uint32_t lookback(uint64_t *state, int tile, uint32_t count, uint32_t *status) {
  const int lane = threadIdx.x & 31;
  if (tile == 0) {
    if (lane == 0) st_relaxed(state, kTilePre | count);
    return 0;
  }
  if (lane == 0) st_relaxed(state + tile, kTileAgg | count);
  uint32_t before = 0;
  for (int j = tile - 1;; j -= 32) {
    const int k = j - lane;  // lane l reads the l-th nearest unread predecessor
    uint64_t v = k >= 0 ? ld_relaxed(state + k) : kTilePre;
    const uint64_t t0 = global_ns();
    for (uint32_t it = 0; __any_sync(kFull, v == 0); ++it) {
      if (v == 0) v = ld_relaxed(state + k);
      if ((it & 63u) == 63u && (ld_acquire(status) & kDevTimeout || global_ns() - t0 > 1000000000ull)) {
        atomicOr(status, kDevTimeout);
        v = v ? v : kTilePre;  // give up: the result is flagged invalid
      }
    }
    const unsigned pre = __ballot_sync(kFull, (v >> 62) == 2);
    const int stop = pre ? __ffs(pre) - 1 : 31;  // the nearest inclusive prefix ends the look-back
    before += __reduce_add_sync(kFull, lane <= stop ? (uint32_t)v : 0u);
    if (pre) break;
  }
  if (lane == 0) st_relaxed(state + tile, kTilePre | (before + count));
  return before;
}

// CTA-wide exclusive scan of one count per thread (256 threads); returns the
// thread's offset and the CTA total in `total`. Ends with a barrier.
__device__ __forceinline__ uint32_t cta_exclusive_scan(uint32_t c, uint32_t *s_warp, uint32_t &total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inc = c;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t v = __shfl_up_sync(kFull, inc, d);
    if (lane >= d) inc += v;
  }
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  uint32_t before = 0;
  total = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    const uint32_t t = s_warp[w];
    before += w < warp ? t : 0u;
    total += t;
  }
  __syncthreads();  // s_warp is reused by the caller
  return before + inc - c;
}

}  // namespace mptc
