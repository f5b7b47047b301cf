// Ordered compactions of a frame: the wavefront order of its blocks, the pending
// list of an inter frame and the unique palette.
#pragma once
#include <cstdint>

#include "lookback.cuh"

namespace mptc {

// Wavefront order of the intra dataflow. Block (x, y) reads, in this frame,
// only blocks of rows y-2sa+1 .. y-1 with columns up to x+sa-1 and blocks of
// row y left of x; with t = x + sa*y every such block has a smaller t. Blocks
// are therefore ranked by (t, y): order[rank] = block index. Blocks of equal t
// never read each other.
__global__ void __launch_bounds__(256) wavefront_order_kernel(int bw, int bh, int sa, uint32_t *__restrict__ order) {
  const int n = bw * bh;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += gridDim.x * blockDim.x) {
    const int y = idx / bw, x = idx - y * bw;
    const long long t = (long long)x + (long long)sa * y;
    long long rank = 0;
    for (int yy = 0; yy < bh; ++yy) {  // blocks with t' < t: x' < t - sa*y'
      const long long c = t - (long long)sa * yy;
      if (c <= 0) break;
      rank += c < bw ? c : bw;
    }
    for (int yy = 0; yy < y; ++yy) {  // blocks with t' == t and y' < y
      const long long xp = t - (long long)sa * yy;
      rank += (xp >= 0 && xp < bw);
    }
    order[rank] = (uint32_t)idx;
  }
}

// Inter frames: the blocks the inter pass left open (done == 0) in wavefront
// order, into pending[0 .. *n_pending); for the fixed-point sweeps each open
// block's first estimate is its stb word (cur[idx]) and the first n_flags
// change flags read (1, 0, 0, ...).
__global__ void __launch_bounds__(256) pending_scan_kernel(const uint32_t *__restrict__ order,
                                                           const uint64_t *__restrict__ done,
                                                           const uint64_t *__restrict__ stb, int n, int ntiles,
                                                           uint64_t *state, uint32_t *claim,
                                                           uint32_t *__restrict__ pending,
                                                           uint32_t *__restrict__ n_pending,
                                                           uint32_t *__restrict__ cur, uint32_t *__restrict__ changed,
                                                           int n_flags, uint32_t *status) {
  depend();
  release_next();
  __shared__ int s_tile;
  __shared__ uint32_t s_warp[8], s_before;
  if (threadIdx.x == 0) s_tile = (int)atomicAdd(claim, 1u);
  __syncthreads();
  const int tile = s_tile, i0 = tile * kScanTile + 4 * threadIdx.x;
  uint32_t blk[4];
  unsigned open = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = i0 + q;
    blk[q] = i < n ? __ldg(order + i) : 0u;
    if (i < n && __ldcg(done + blk[q]) == 0ull) open |= 1u << q;
  }
  uint32_t total;
  uint32_t off = cta_exclusive_scan(__popc(open), s_warp, total);
  if (threadIdx.x < 32) {
    const uint32_t b = lookback(state, tile, total, status);
    if (threadIdx.x == 0) s_before = b;
  }
  __syncthreads();
  off += s_before;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if ((open >> q) & 1u) {
      pending[off++] = blk[q];
      cur[blk[q]] = (uint32_t)(__ldg(stb + blk[q]) >> 32);
    }
  if (tile == ntiles - 1 && threadIdx.x == 0) *n_pending = s_before + total;
  if (tile == 0)
    for (int f = threadIdx.x; f < n_flags; f += blockDim.x) changed[f] = f == 0 ? 1u : 0u;
}

// ----------------------------------------------------------------- unique --
// The unique palette lists the stb interp of every unaccepted block in raster
// order (codec/dxt_image.cpp:953-954), compacted in one pass; the same pass
// counts the frame's inter, intra and unique blocks into stats[0..2].
__global__ void __launch_bounds__(256) unique_scan_kernel(const uint16_t *__restrict__ motion,
                                                          const uint64_t *__restrict__ stb, int nblk, int ntiles,
                                                          uint64_t *state, uint32_t *claim,
                                                          uint32_t *__restrict__ unique,
                                                          uint32_t *__restrict__ n_unique,
                                                          uint32_t *__restrict__ stats, uint32_t *status) {
  depend();
  release_next();
  __shared__ int s_tile;
  __shared__ uint32_t s_warp[8], s_before;
  if (threadIdx.x == 0) s_tile = (int)atomicAdd(claim, 1u);
  __syncthreads();
  const int tile = s_tile, i0 = tile * kScanTile + 4 * threadIdx.x;
  unsigned uq = 0;
  int ni = 0, na = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = i0 + q;
    if (i < nblk) {
      const uint16_t m = motion[i];
      if (m == 0xFFFFu)
        uq |= 1u << q;
      else if (m & 0x80u)
        ++ni;
      else
        ++na;
    }
  }
  uint32_t total;
  uint32_t off = cta_exclusive_scan(__popc(uq), s_warp, total);
  ni = __reduce_add_sync(kFull, ni);
  na = __reduce_add_sync(kFull, na);
  if ((threadIdx.x & 31) == 0) {
    if (ni) atomicAdd(stats + 0, (uint32_t)ni);
    if (na) atomicAdd(stats + 1, (uint32_t)na);
  }
  if (threadIdx.x < 32) {
    const uint32_t b = lookback(state, tile, total, status);
    if (threadIdx.x == 0) {
      s_before = b;
      if (total) atomicAdd(stats + 2, total);
    }
  }
  __syncthreads();
  off += s_before;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if ((uq >> q) & 1u) unique[off++] = (uint32_t)(__ldg(stb + i0 + q) >> 32);
  if (tile == ntiles - 1 && threadIdx.x == 0) *n_unique = s_before + total;
}

}  // namespace mptc
