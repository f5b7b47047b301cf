// InterBlockSearch (codec/dxt_image.cpp:715-774): the run search for sa <= 8 with
// the overflow search of noisy runs, and the search of wider windows.
#pragma once
#include <cstdint>

#include "completion.cuh"

namespace mptc {

// ------------------------------------------------------------------ inter --
// InterBlockSearch, codec/dxt_image.cpp:715-774: rows j = by-sa .. by+sa-1,
// columns i = bx-sa .. bx+sa-1 (both ascending); motion (i-bx+sa)|0x80,
// (j-by+sa)|0x80. Accepted blocks become final here; the others are left for
// the intra pass (done = 0).
// Refit, validity and error depend only on the block and the candidate index
// word, so positions holding equal words get equal results, and each distinct
// word of the window is evaluated once: on smooth content a 16x16 window holds
// few distinct words (about 15% of the positions on the 1080p test stream).

// ------------------------------------------------------------ inter runs --
// The search for sa <= 8, one warp per run of up to kRun horizontally
// adjacent blocks of a row. Their windows share all rows and overlap in all but
// a few columns, so the warp deduplicates the union of the windows (w2 rows of
// at most w2 + kRun - 1 columns, a row at a time, lane = column) once, recording
// for each distinct word the union columns where it occurs (a bit mask). The
// pairs of a block and a distinct word of its window (other than its own) are
// queued and evaluated 32 at a time across the blocks, so that the lanes stay
// busy although a window holds some 33 words: refit_quick for each, refit_exact
// for the few that it leaves out, queued until they fill a pass. Each result is
// kept as a 16-bit rank per block and word. Per block the reference's selection
// is then one minimum over the window's positions, the smallest rank at its
// first position; only where a window holds an err_diff < 0 (12-19% of the
// blocks) further passes find the first err_diff <= 0 and an err_diff < 0 in a
// later row. The selected words of all blocks are refitted once more together
// for their endpoints.
// The hash table's empty marker is the first block's own word, which keeps a
// dedicated slot 0 outside the table. The blocks of a run whose union holds more
// than kRunWords distinct words (noisy content) are appended to a list that
// inter_overflow_kernel searches afterwards with a CTA per block: those runs
// cost several times a smooth one and, kept in one warp, would hold their SM
// long after the other warps finished.
// Bound by issue (80% of the slots), 846 warp instructions a block on the 1080p
// test stream: evaluation about 255, deduplication 194, lists 89, selection 67, the
// exact refits about 70, the rest staging. 122 us a frame, against 226 (1,566
// instructions) with each block's words evaluated by themselves from a table of
// float products in shared memory.
constexpr int kRun = 8;
constexpr int kRunWords = 128;  // distinct union words handled by the run table
constexpr int kRunBuckets = 256;
__device__ __forceinline__ uint32_t run_hash(uint32_t v) { return (v * 2654435761u) >> 24; }
// err_diff e as a rank: 0 for e < 0, e + 1 for the others (err_diffs are at most
// 65025), kNoRank where the refit would swap the endpoints
constexpr uint32_t kNoRank = 0xFFFFu;

struct RunTab {
  static constexpr int kSlotBits = 8;  // of a pair's word; its block above them
  static constexpr int kCols = 16 + kRun - 1;  // union columns at sa = 8
  static constexpr int kStride = kCols + 1;
  // the marker, kRunWords words, and the up to kCols further new words of the
  // row that crosses the limit
  static constexpr int kSlots = 1 + kRunWords + kCols;
  static constexpr int kSentinel = kSlots;  // slot of out-of-frame positions
  PixBlocks<kRun> px;
  int orig[kRun];
  uint32_t own[kRun];
  union {
    struct {
      uint32_t bkey[kRunBuckets];  // word, or the marker when empty
      uint8_t bslot[kRunBuckets];
    };
    struct {  // pairs to evaluate: block << 8 | slot
      uint16_t quick[32 + 32 * kRun], exact[64];
    };
  };
  uint32_t key[kSlots];
  uint32_t cols[kSlots];           // union columns holding the word (bit per column)
  uint32_t at[kSlots];             // a block of the previous frame holding the word
  uint8_t pslot[16 * kStride];     // slot of each union position
  union {
    uint32_t word[16][kCols];               // the union's words while they are inserted
    uint16_t rank[kRun][kSlots + 1];  // of each block and word
  };
};

// Evaluates a pair of a run from the integer sums; false where run_exact has to.
template <class Tab>
__device__ __forceinline__ bool run_quick(const Tab &rt, const float4 *wdesc, const SnapTables &st, uint32_t pair,
                                          int &e) {
  const int k = (int)(pair >> Tab::kSlotBits), s = (int)(pair & ((1u << Tab::kSlotBits) - 1u));
  const float4 d = __ldg(wdesc + rt.at[s]);
  const WeightSums ws{d.x, d.y, d.z, d.w};
  RefitValues r;
  uint32_t eps;
  const bool ok = refit_quick(PixBlock<kRun>{rt.px, k}, st, rt.key[s], ws, r);
  e = refit_error(PixBlock<kRun>{rt.px, k}, r, rt.key[s], rt.orig[k], eps);
  return ok;
}
// Evaluates a pair by the reference's own steps: its err_diff and endpoints.
template <class Tab>
__device__ __forceinline__ uint2 run_exact(const Tab &rt, const float4 *wdesc, const SnapTables &st, uint32_t pair) {
  const int k = (int)(pair >> Tab::kSlotBits), s = (int)(pair & ((1u << Tab::kSlotBits) - 1u));
  const float4 d = __ldg(wdesc + rt.at[s]);
  const WeightSums ws{d.x, d.y, d.z, d.w};
  RefitValues r;
  uint32_t eps;
  refit_exact(PixBlock<kRun>{rt.px, k}, st, rt.key[s], ws, r);
  const int e = refit_error(PixBlock<kRun>{rt.px, k}, r, rt.key[s], rt.orig[k], eps);
  return make_uint2((uint32_t)e, eps);
}
// Pair q of a run for refit_by_channels.
template <class Tab>
__device__ __forceinline__ ExactCase<kRun> run_case(const Tab &rt, const float4 *wdesc, uint32_t pair) {
  const int k = (int)(pair >> Tab::kSlotBits), s = (int)(pair & ((1u << Tab::kSlotBits) - 1u));
  return ExactCase<kRun>{PixBlock<kRun>{rt.px, k}, rt.key[s], __ldg(wdesc + rt.at[s]), rt.orig[k]};
}
__device__ __forceinline__ uint16_t run_rank(int e) {
  return (uint16_t)(e == kInvalid ? kNoRank : (uint32_t)max(e, -1) + 1u);
}

// Block k's row of pixels (load_channels) into px by four adjacent lanes, lane r of
// them row r; every lane of the warp calls it, `store` where its block exists.
template <int N>
__device__ __forceinline__ void stage_row(PixBlocks<N> &px, int k, uint32_t c0, uint32_t c1, uint32_t c2, int r,
                                          bool store) {
  uint32_t s0 = __dp4a(c0, 0x01010101u, 0u), s1 = __dp4a(c1, 0x01010101u, 0u), s2 = __dp4a(c2, 0x01010101u, 0u);
  uint32_t sq = __dp4a(c0, c0, __dp4a(c1, c1, __dp4a(c2, c2, 0u)));
#pragma unroll
  for (int o = 1; o <= 2; o <<= 1) {
    s0 += __shfl_xor_sync(kFull, s0, o);
    s1 += __shfl_xor_sync(kFull, s1, o);
    s2 += __shfl_xor_sync(kFull, s2, o);
    sq += __shfl_xor_sync(kFull, sq, o);
  }
  if (store) {
    px.w[0][k][r] = c0;
    px.w[1][k][r] = c1;
    px.w[2][k][r] = c2;
    if (r == 0) *reinterpret_cast<uint4 *>(px.w[3][k]) = make_uint4(s0, s1, s2, sq);
  }
}

// The pixels of a run's nb blocks by one warp, one block row per lane.
__device__ __forceinline__ void stage_run(PixBlocks<kRun> &px, const SearchParams &P, int bx0, int by, int nb, int lane) {
  const int k = lane >> 2, r = lane & 3;
  uint32_t c0 = 0, c1 = 0, c2 = 0;
  if (k < nb) load_channels(P.rgb, P.width, bx0 + k, 4 * by + r, c0, c1, c2);
  stage_row(px, k, c0, c1, c2, r, k < nb);
}

// SA: the search area when fixed at compile time (its constants fold), 0 to
// read it from P. A persistent grid: each warp takes the next unit of work
// from *next_run (zero at launch), which keeps all warps busy to the end
// although runs differ in cost. run: blocks per run, at most RUN.
template <int WARPS, int RUN, int SA>
__global__ void __launch_bounds__(WARPS * 32, 32 / WARPS)
    inter_run_kernel(SearchParams P, uint32_t *next_run, int run, uint32_t *ovf_count, uint32_t *ovf_list) {
  using Tab = RunTab;
  static_assert(RUN == kRun && 4 * kRun == 32, "a run's block rows take one lane each");
  static_assert(Tab::kSentinel <= 255 && Tab::kSlots - 1 <= kRunBuckets, "slots are bytes; buckets hold the words");
  __shared__ Tab s_run[WARPS];
  __shared__ SnapTables s_snap;
  build_snap_edges(s_snap);
  __syncthreads();
  depend();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Tab &rt = s_run[warp];
  const unsigned lt_mask = (1u << lane) - 1u;
  const int sa = SA ? SA : P.sa;
  const int w2 = 2 * sa;
  const uint32_t *prev_hi = reinterpret_cast<const uint32_t *>(P.prev) + 1;
  for (;;) {
    int unit = 0;
    if (lane == 0) unit = (int)atomicAdd(next_run, 1u);
    unit = __shfl_sync(kFull, unit, 0);
    const int per_row = (P.bw + run - 1) / run, by = unit / per_row;
    if (by >= P.bh) break;
    const int bx0 = (unit - by * per_row) * run, nb = min(run, P.bw - bx0);
    const int j0 = by - sa, i0 = bx0 - sa;
    const uint32_t marker = (uint32_t)(P.stb[by * P.bw + bx0] >> 32);
    for (int b = lane; b < kRunBuckets / 4; b += 32)
      reinterpret_cast<uint4 *>(rt.bkey)[b] = make_uint4(marker, marker, marker, marker);
    if (lane < nb) {
      rt.orig[lane] = P.orig_err[by * P.bw + bx0 + lane];
      rt.own[lane] = (uint32_t)(P.stb[by * P.bw + bx0 + lane] >> 32);
    }
    // the union's words, all loads first so their latencies overlap
    const bool col_in = lane < w2 + nb - 1 && i0 + lane >= 0 && i0 + lane < P.bw;
    const unsigned colm = __ballot_sync(kFull, col_in);
    if (lane < Tab::kCols) {
#pragma unroll
      for (int r = 0; r < 16; ++r)
        if (r < w2) {
          const int j = j0 + r;
          rt.word[r][lane] = col_in && j >= 0 && j < P.bh ? __ldg(prev_hi + 2 * (size_t)(j * P.bw + i0 + lane)) : marker;
        }
    }
    __syncwarp();
    stage_run(rt.px, P, bx0, by, nb, lane);
    // the distinct words, row by row: a word's first lane looks it up
    int nuniq = 1;
    uint32_t mark_cols = 0, mark_at = 0;  // the marker's
    bool overflow = false;
#pragma unroll 1
    for (int r = 0; r < w2; ++r) {
      const int j = j0 + r;
      int slot = Tab::kSentinel;
      if (j >= 0 && j < P.bh) {  // warp-uniform
        const uint32_t cand = lane < Tab::kCols ? rt.word[r][lane] : marker;
        const unsigned peers = __match_any_sync(kFull, cand) & colm;
        bool is_new = false;
        uint32_t b = 0;
        slot = 0;
        if (cand == marker) {
          mark_cols |= peers;
          if (peers) mark_at = (uint32_t)(j * P.bw + i0 + __ffs(peers) - 1);
        } else if (lane == __ffs(peers) - 1) {
          b = run_hash(cand);
          uint32_t old;
          while ((old = atomicCAS(&rt.bkey[b], marker, cand)) != marker && old != cand)
            b = (b + 1) & (kRunBuckets - 1);  // ends: at most kSlots - 1 words in kRunBuckets
          is_new = old == marker;
          if (!is_new) {  // inserted by an earlier row
            slot = rt.bslot[b];
            rt.cols[slot] |= peers;
          }
        }
        const unsigned newm = __ballot_sync(kFull, is_new);
        if (is_new) {
          slot = nuniq + __popc(newm & lt_mask);
          rt.bslot[b] = (uint8_t)slot;
          rt.key[slot] = cand;
          rt.cols[slot] = peers;
          rt.at[slot] = (uint32_t)(j * P.bw + i0 + lane);
        }
        slot = __shfl_sync(kFull, slot, max(__ffs(peers) - 1, 0));
        if (!col_in) slot = Tab::kSentinel;
        nuniq += __popc(newm);
        __syncwarp();  // this row's slot writes land before later rows read them
      }
      if (lane < Tab::kCols) rt.pslot[r * Tab::kStride + lane] = (uint8_t)slot;
      if (nuniq > 1 + kRunWords) {  // warp-uniform
        overflow = true;
        break;
      }
    }
    if (overflow) {
      if (lane == 0) {
        const uint32_t at = atomicAdd(ovf_count, (uint32_t)nb);
        for (int k = 0; k < nb; ++k) ovf_list[at + k] = (uint32_t)(by * P.bw + bx0 + k);
      }
      __syncwarp();
      continue;
    }
    {  // the marker's lanes (a word's peers are the same row by row, its lanes are not)
      const uint32_t c = __reduce_or_sync(kFull, mark_cols), at = __reduce_max_sync(kFull, mark_at);
      if (lane == 0) {
        rt.key[0] = marker;
        rt.cols[0] = c;
        rt.at[0] = at;
      }
    }
    __syncwarp();
    // the pairs, queued and evaluated
    int nquick = 0, nexact = 0;
#pragma unroll 1
    for (int s0 = 0; s0 < nuniq; s0 += 32) {
      const int s = s0 + lane;
      // the blocks whose window holds the word: bit k, columns k .. k + w2 - 1
      uint32_t take = 0;
      if (s < nuniq) {
        take = rt.cols[s];
        if (SA == 8) {
          take |= take >> 1;
          take |= take >> 2;
          take |= take >> 4;
          take |= take >> 8;
        } else {
          const uint32_t c = take;
          for (int i = 1; i < w2; ++i) take |= c >> i;
        }
        take &= (1u << nb) - 1u;
        const uint32_t key = rt.key[s];
        uint32_t own = 0;
#pragma unroll
        for (int k = 0; k < kRun; ++k) own |= key == rt.own[k] ? 1u << k : 0u;
        for (own &= take; own; own &= own - 1u) {  // the block's own word: err_diff 0, no refit
          const int k = __ffs(own) - 1;
          rt.rank[k][s] = 1u;
          take &= ~(1u << k);
        }
      }
      int at = __popc(take);
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(kFull, at, d);
        if (lane >= d) at += v;
      }
      const int total = __shfl_sync(kFull, at, 31);
      at += nquick - __popc(take);
#pragma unroll
      for (int k = 0; k < kRun; ++k)
        if ((take >> k) & 1u) rt.quick[at++] = (uint16_t)((k << 8) | s);
      nquick += total;
      __syncwarp();
      const bool last = s0 + 32 >= nuniq;
      while (nquick >= 32 || (last && nquick + nexact > 0)) {
        // full passes from the queues' ends; what is left with the last words
        if (nquick >= 32 || (last && nquick > 0)) {
          const int n = min(nquick, 32);
          nquick -= n;
          bool out = false;
          uint32_t pair = 0;
          if (lane < n) {
            pair = rt.quick[nquick + lane];
            int e;
            out = !run_quick(rt, P.wdesc, s_snap, pair, e);
            rt.rank[pair >> 8][pair & 255u] = run_rank(e);
          }
          const unsigned om = __ballot_sync(kFull, out);
          if (out) rt.exact[nexact + __popc(om & lt_mask)] = (uint16_t)pair;
          nexact += __popc(om);
          __syncwarp();
        }
        if (last && nquick == 0 && nexact > 0 && nexact <= kByChannels) {
          const int n = nexact;
          nexact = 0;
          const uint2 x =
              refit_by_channels(s_snap, n, lane, [&](int q) { return run_case(rt, P.wdesc, rt.exact[q]); });
          if (lane < n) {
            const uint32_t pair = rt.exact[lane];
            rt.rank[pair >> 8][pair & 255u] = run_rank((int)x.x);
          }
          __syncwarp();
        } else if (nexact >= 32 || (last && nquick == 0 && nexact > 0)) {
          const int n = min(nexact, 32);
          nexact -= n;
          if (lane < n) {
            const uint32_t pair = rt.exact[nexact + lane];
            rt.rank[pair >> 8][pair & 255u] = run_rank((int)run_exact(rt, P.wdesc, s_snap, pair).x);
          }
          __syncwarp();
        }
      }
    }
    if (lane < nb) rt.rank[lane][Tab::kSentinel] = (uint16_t)kNoRank;
    __syncwarp();
    // lane k: its block's selected position + 1 (0: none) << 8 | slot
    uint32_t win = 0;
#pragma unroll 1
    for (int k = 0; k < nb; ++k) {
      const uint16_t *rank = rt.rank[k];
      const uint8_t *pslot = rt.pslot + k;
      // rank << 8 | position, in scan order (rows, then columns)
      uint32_t best = 0xFFFFFFFFu;
      auto each = [&](auto f) {
        if (SA == 8) {
          const uint8_t *at = pslot + (lane >> 4) * Tab::kStride + (lane & 15);
#pragma unroll
          for (int c = 0; c < 8; ++c) f(rank[at[2 * c * Tab::kStride]], (uint32_t)(32 * c + lane));
        } else {
#pragma unroll 1
          for (int p = lane; p < w2 * w2; p += 32) f(rank[pslot[p / w2 * Tab::kStride + p % w2]], (uint32_t)p);
        }
      };
      each([&](uint32_t v, uint32_t p) { best = min(best, (v << 8) | p); });
      best = __reduce_min_sync(kFull, best);
      int pos = -1;
      if (best < 256u) {  // an err_diff < 0
        if (P.thr >= 0) {
          uint32_t first = 256u;
          int last = -1;
          each([&](uint32_t v, uint32_t p) {
            if (v <= 1u) first = min(first, p);
            if (v == 0u) last = max(last, (int)((p / (uint32_t)w2 << 8) | (255u - p)));
          });
          first = __reduce_min_sync(kFull, first);
          last = __reduce_max_sync(kFull, last);
          pos = (last >> 8) > (int)(first / (uint32_t)w2) ? 255 - (last & 255) : (int)first;
        }
      } else if (best < kNoRank << 8 && (int)(best >> 8) - 1 <= P.thr) {
        pos = (int)(best & 255u);
      }
      if (lane == k && pos >= 0)
        win = ((uint32_t)pos + 1u) << 8 | pslot[pos / w2 * Tab::kStride + pos % w2];
    }
    // the selected words' endpoints (a block's own word needs none: computed, unused)
    if (lane < nb) rt.exact[lane] = (uint16_t)((uint32_t)lane << 8 | (win & 255u));
    __syncwarp();
    const uint2 refit =
        refit_by_channels(s_snap, nb, lane, [&](int q) { return run_case(rt, P.wdesc, rt.exact[q]); });
    if (lane < nb) {
      const int idx = by * P.bw + bx0 + lane;
      uint64_t word = 0;
      if (win != 0u) {
        const uint32_t s = win & 255u, pos = (win >> 8) - 1u;
        uint64_t blk = P.stb[idx];
        if (rt.key[s] != rt.own[lane]) blk = (uint64_t)refit.y | ((uint64_t)rt.key[s] << 32);
        const uint32_t row = pos / (uint32_t)w2, col = pos - row * (uint32_t)w2;
        P.final_blk[idx] = blk;
        P.motion[idx] = (uint16_t)((col | 0x80) | ((row | 0x80) << 8));
        word = done_word(blk);
      }
      P.done[idx] = word;
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------ wide windows --
// The search for sa > 8, one CTA per run of up to kRun adjacent blocks: the same
// three parts as a run of inter_run_kernel, over the union of the run's windows,
// w2 rows of w2 + kRun - 1 columns (up to 126 x 133), by eight warps.
// 1. Every position's word is looked up in a hash table in shared memory, a
//    compare-and-swap only where a plain read finds an empty bucket, and the
//    position keeps the bucket.
// 2. Every pair of a block and a distinct word is evaluated (words at the
//    union's edges also for the blocks whose window they miss, which no position
//    then selects): a warp takes 32 words of one block, refit_quick, the near ties
//    queued for refit_exact. Results are 16-bit ranks by block and bucket.
// 3. A warp per block takes the reference's selection over the window's
//    positions, and one warp refits the selected words for their endpoints.
// A union of more distinct words than the table takes (noise) is searched in
// slabs of rows that fit it, whose selections are merged.
// A warp per block and a table per span of 256 positions before: 510 us for an
// 856x480 frame at sa 24, 184 now (the whole frame 306, before 690).
constexpr int kWideThreads = 256, kWideBuckets = 1024, kWideWords = 640;
// The buckets' table is never full: a thread inserts only after it has read a
// count of at most kWideWords, and counts each word before its next.
static_assert(kWideWords + kWideThreads < kWideBuckets, "a probe ends at an empty bucket");
static_assert(kWideWords >= 126 + kRun - 1, "a row of any union fits");

struct WideTab {
  static constexpr int kSlotBits = 11;
  static constexpr int kMark = kWideBuckets;      // slot of the empty buckets' word, the first block's own
  static constexpr int kNone = kWideBuckets + 1;  // slot of out-of-frame positions
  PixBlocks<kRun> px;
  int orig[kRun];
  uint32_t own[kRun];
  uint32_t key[kWideBuckets + 1];
  uint32_t at[kWideBuckets + 1];  // a block of the previous frame holding the word
  uint16_t list[kWideBuckets];    // the used buckets
  uint16_t rank[kRun][kWideBuckets + 2];
  uint16_t exact[kWideThreads / 32][64];  // a warp's near ties: block << kSlotBits | slot
  int win[kRun];                  // selected position (-1: none)
  int n;                          // used buckets
};
// The dynamic shared memory: the table and a 16-bit slot per union position.
__host__ __device__ constexpr int wide_smem(int sa) {
  return (int)sizeof(WideTab) + 2 * (2 * sa) * (2 * sa + kRun - 1);
}

__global__ void __launch_bounds__(kWideThreads, 4) inter_wide_kernel(SearchParams P, int run) {
  extern __shared__ __align__(16) uint8_t wide_mem[];
  __shared__ SnapTables s_snap;
  WideTab &wt = *reinterpret_cast<WideTab *>(wide_mem);
  uint16_t *pslot = reinterpret_cast<uint16_t *>(wide_mem + sizeof(WideTab));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt_mask = (1u << lane) - 1u;
  constexpr int kWarps = kWideThreads / 32;
  build_snap_edges(s_snap);
  depend();
  const int per_row = (P.bw + run - 1) / run, by = blockIdx.x / per_row;
  const int bx0 = (blockIdx.x - by * per_row) * run, nb = min(run, P.bw - bx0);
  const int sa = P.sa, w2 = 2 * sa, cols = w2 + nb - 1, j0 = by - sa, i0 = bx0 - sa;
  const uint32_t *prev_hi = reinterpret_cast<const uint32_t *>(P.prev) + 1;
  const uint32_t marker = (uint32_t)(P.stb[by * P.bw + bx0] >> 32);
  if (warp == 0) {
    if (lane < nb) {
      wt.orig[lane] = P.orig_err[by * P.bw + bx0 + lane];
      wt.own[lane] = (uint32_t)(P.stb[by * P.bw + bx0 + lane] >> 32);
      wt.rank[lane][WideTab::kNone] = (uint16_t)kNoRank;
    }
    stage_run(wt.px, P, bx0, by, nb, lane);
  }
  volatile uint32_t *key = wt.key;
  volatile int *count = &wt.n;
  // warp k: its block's selection so far (see LaneSel): the smallest rank at its first
  // position, the first err_diff <= 0, an err_diff < 0 in the last row that holds one
  uint32_t best = 0xFFFFFFFFu, first = 1u << 14;
  int last = -1;
  int slab = w2;  // rows at a time
  for (int r0 = 0; r0 < w2;) {
    const int r1 = min(w2, r0 + slab);
    __syncthreads();  // the previous slab's readers are done
    for (int b = tid; b <= kWideBuckets; b += kWideThreads) wt.key[b] = marker;
    if (tid == 0) {
      wt.n = 0;
      wt.at[WideTab::kMark] = ~0u;
    }
    __syncthreads();
    // 1. the distinct words
    for (int r = r0 + warp; r < r1; r += kWarps) {
      if (__any_sync(kFull, *count > kWideWords)) break;
      const int j = j0 + r;
      const bool row_in = j >= 0 && j < P.bh;
      const uint32_t *src = prev_hi + 2 * ((ptrdiff_t)j * P.bw + i0);
      auto in = [&](int c) { return row_in && c < cols && i0 + c >= 0 && i0 + c < P.bw; };
      uint32_t next = in(lane) ? __ldg(src + 2 * lane) : marker;
#pragma unroll 1
      for (int c = lane; c < cols + lane; c += 32) {  // the warp's lanes together
        const uint32_t cand = next;
        if (in(c + 32)) next = __ldg(src + 2 * (c + 32));
        if (c >= cols) continue;
        uint32_t slot = WideTab::kNone;
        if (in(c)) {
          const uint32_t nidx = (uint32_t)(j * P.bw + i0 + c);
          if (cand == marker) {
            slot = WideTab::kMark;
            wt.at[WideTab::kMark] = nidx;  // any of them
          } else {
            uint32_t b = (cand * 2654435761u) >> 22;
            for (;;) {
              uint32_t old = key[b];
              if (old == marker) {
                if (*count > kWideWords) break;  // the slab is given up
                old = atomicCAS(&wt.key[b], marker, cand);
                if (old == marker) {
                  wt.at[b] = nidx;
                  wt.list[atomicAdd(&wt.n, 1)] = (uint16_t)b;
                  old = cand;
                }
              }
              if (old == cand) break;
              b = (b + 1) & (kWideBuckets - 1);
            }
            slot = b;
          }
        }
        pslot[(r - r0) * cols + c] = (uint16_t)slot;
      }
      __syncwarp();
    }
    __syncthreads();
    const int used = wt.n;
    if (used > kWideWords) {  // only a slab of more rows than this, which always fit
      slab = kWideWords / cols;
      continue;
    }
    // 2. the pairs
    {
      const int total = used + (wt.at[WideTab::kMark] != ~0u ? 1 : 0), chunks = (total + 31) / 32;
      uint16_t *queue = wt.exact[warp];
      int queued = 0;
      auto drain = [&](int n) {
        queued -= n;
        if (lane < n) {
          const uint32_t pair = queue[queued + lane];
          wt.rank[pair >> WideTab::kSlotBits][pair & ((1u << WideTab::kSlotBits) - 1u)] =
              run_rank((int)run_exact(wt, P.wdesc, s_snap, pair).x);
        }
        __syncwarp();
      };
#pragma unroll 1
      for (int t = warp; t < nb * chunks; t += kWarps) {
        const int c = t / nb, k = t - c * nb, i = 32 * c + lane;
        bool out = false;
        uint32_t pair = 0;
        if (i < total) {
          const uint32_t s = i < used ? wt.list[i] : WideTab::kMark;
          pair = (uint32_t)k << WideTab::kSlotBits | s;
          int e = 0;  // the block's own word: err_diff 0, no refit
          if (wt.key[s] != wt.own[k]) out = !run_quick(wt, P.wdesc, s_snap, pair, e);
          wt.rank[k][s] = run_rank(e);
        }
        const unsigned om = __ballot_sync(kFull, out);
        if (out) queue[queued + __popc(om & lt_mask)] = (uint16_t)pair;
        queued += __popc(om);
        __syncwarp();
        if (queued >= 32) drain(32);
      }
      if (queued > kByChannels) {
        drain(queued);
      } else if (queued > 0) {
        const uint2 x = refit_by_channels(s_snap, queued, lane, [&](int q) { return run_case(wt, P.wdesc, queue[q]); });
        if (lane < queued) {
          const uint32_t pair = queue[lane];
          wt.rank[pair >> WideTab::kSlotBits][pair & ((1u << WideTab::kSlotBits) - 1u)] = run_rank((int)x.x);
        }
      }
    }
    __syncthreads();
    // 3. the selections
    if (warp < nb) {
      const uint16_t *rank = wt.rank[warp], *mine = pslot + warp;
      const int p0 = r0 * w2, npos = (r1 - r0) * w2, drow = 32 / w2, dcol = 32 - drow * w2;
      const int row0 = lane / w2, col0 = lane - row0 * w2;
      auto each = [&](auto f) {
        int at = row0 * cols + col0, col = col0;
#pragma unroll 4
        for (int p = lane; p < npos; p += 32) {
          f((uint32_t)rank[mine[at]], (uint32_t)(p0 + p));
          at += drow * cols + dcol;
          col += dcol;
          if (col >= w2) {
            col -= w2;
            at += cols - w2;
          }
        }
      };
      // rank << 14 | position, in scan order (rows, then columns)
      uint32_t b = 0xFFFFFFFFu;
      each([&](uint32_t v, uint32_t p) { b = min(b, (v << 14) | p); });
      b = __reduce_min_sync(kFull, b);
      if (b < 1u << 14) {  // an err_diff < 0
        each([&](uint32_t v, uint32_t p) {
          if (v <= 1u) first = min(first, p);
          if (v == 0u) last = max(last, (int)((p / (uint32_t)w2 << 14) | (16383u - p)));
        });
      } else if (b < 2u << 14) {  // an err_diff of 0, the first of this slab
        first = min(first, b & 16383u);
      }
      best = min(best, b);
    }
    r0 = r1;
  }
  if (warp < nb) {
    int pos = -1;
    if (best < 2u << 14) {
      first = __reduce_min_sync(kFull, first);
      last = __reduce_max_sync(kFull, last);
      if (P.thr >= 0) pos = last >= 0 && (last >> 14) > (int)(first / (uint32_t)w2) ? 16383 - (last & 16383) : (int)first;
    } else if (best < kNoRank << 14 && (int)(best >> 14) - 1 <= P.thr) {
      pos = (int)(best & 16383u);
    }
    if (lane == 0) wt.win[warp] = pos;
  }
  __syncthreads();
  if (warp != 0) return;
  // the selected words' endpoints (a block's own word needs none: computed, unused);
  // each word in a slot of the table
  const int pos = lane < nb ? wt.win[lane] : -1, row = max(pos, 0) / w2, col = max(pos, 0) - row * w2;
  uint32_t cand = marker;
  if (pos >= 0) {
    const uint32_t nidx = (uint32_t)((j0 + row) * P.bw + i0 + lane + col);
    cand = __ldg(prev_hi + 2 * (size_t)nidx);
    wt.at[lane] = nidx;
  } else if (lane < nb) {
    wt.at[lane] = 0;
  }
  if (lane < nb) wt.key[lane] = cand;
  __syncwarp();
  const uint2 refit = refit_by_channels(s_snap, nb, lane, [&](int q) {
    return run_case(wt, P.wdesc, (uint32_t)q << WideTab::kSlotBits | (uint32_t)q);
  });
  if (lane < nb) {
    const int idx = by * P.bw + bx0 + lane;
    uint64_t word = 0;
    if (pos >= 0) {
      uint64_t blk = P.stb[idx];
      if (cand != wt.own[lane]) blk = (uint64_t)refit.y | ((uint64_t)cand << 32);
      P.final_blk[idx] = blk;
      P.motion[idx] = (uint16_t)((col | 0x80) | ((row | 0x80) << 8));
      word = done_word(blk);
    }
    P.done[idx] = word;
  }
}

// Weight sums of the refit for every block's index word (the candidates the
// next search reads), one thread per block. As the first kernel of a search it
// also zeroes the frame's work words and, for an intra frame, the completion
// words (zeroed: n of them, or null), instead of a memset each before it.
__global__ void __launch_bounds__(256) weight_desc_kernel(const uint64_t *__restrict__ blocks, int n,
                                                          float4 *__restrict__ desc, uint32_t *__restrict__ work,
                                                          int n_work, uint64_t *__restrict__ zeroed) {
  __shared__ float4 s_wk[4];
  build_weight_table(s_wk);
  __syncthreads();
  depend();
  release_next();
  const int first = blockIdx.x * blockDim.x + threadIdx.x;
  for (int i = first; i < n_work; i += gridDim.x * blockDim.x) work[i] = 0u;
  for (int i = first; i < n; i += gridDim.x * blockDim.x) {
    if (zeroed) zeroed[i] = 0ull;
    const WeightSums w = weight_sums((uint32_t)(__ldg(blocks + i) >> 32), s_wk);
    desc[i] = make_float4(w.asq, w.bsq, w.ab, w.f);
  }
}

// The blocks of the runs whose union overflowed the run table (noisy
// content), list[0 .. *count): one CTA per block and one window position per
// thread (sa <= 8: at most 256 positions), every position evaluated by its
// own thread, then the closed-form selection over the CTA (cta_select). The
// many distinct words of such windows are evaluated side by side instead of
// in a warp's successive rounds.
// One listed block searched by a CTA (THREADS >= 256, sa <= 8): thread t
// evaluates window position t, then the CTA-wide closed-form selection.
// Starts with a barrier (the previous block's readers of s_tab are done).
template <int THREADS>
__device__ __forceinline__ void cta_block_search(const SearchParams &P, int idx, BlockTab &s_tab,
                                                 const uint8_t *s_snap5, const uint8_t *s_snap6,
                                                 CtaReduce<THREADS> &red, int *s_sumsq) {
  const int tid = threadIdx.x, lane = tid & 31;
  const int w2 = 2 * P.sa, npos = w2 * w2;
  const int row = tid / w2, col = tid - row * w2;  // the thread's window position tid
  const uint32_t *prev_hi = reinterpret_cast<const uint32_t *>(P.prev) + 1;
  const int by = idx / P.bw, bx = idx - by * P.bw;
  const uint64_t stb = __ldg(P.stb + idx);
  const uint32_t own = (uint32_t)(stb >> 32);
  __syncthreads();
  if (tid < 32) {
    const int sq = stage_block(s_tab, P.rgb, P.width, bx, by, lane);
    if (tid == 0) *s_sumsq = sq;
  }
  __syncthreads();
  const int orig = __ldg(P.orig_err + idx), sumsq = *s_sumsq;
  const PixelGroups pg = load_groups(s_tab);
  LaneSel ls;
  uint32_t cand = own, eps = 0;
  const int j = by - P.sa + row, i = bx - P.sa + col;
  if (tid < npos && i >= 0 && j >= 0 && i < P.bw && j < P.bh) {
    const size_t nidx = (size_t)j * P.bw + i;
    cand = __ldg(prev_hi + 2 * nidx);
    int e = 0;  // the block's own word: the stb block, no refit
    if (cand != own) {
      const float4 d = __ldg(P.wdesc + nidx);
      const WeightSums ws{d.x, d.y, d.z, d.w};
      int refit = 0;
      e = eval_candidate(s_tab, pg, s_snap5, s_snap6, cand, ws, own, orig, sumsq, eps, refit);
    }
    ls.add(tid, row, e);
  }
  int m, pick;
  const int sel = cta_select<THREADS>(ls, red, w2, m, pick);
  const bool accept = sel >= 0 && m <= P.thr;  // CTA-uniform
  if (accept ? tid == sel : tid == 0) {
    uint64_t word = 0;
    if (accept) {
      const uint64_t blk = cand == own ? stb : ((uint64_t)eps | ((uint64_t)cand << 32));
      P.final_blk[idx] = blk;
      P.motion[idx] = (uint16_t)((col | 0x80) | ((row | 0x80) << 8));
      word = done_word(blk);
    }
    P.done[idx] = word;
  }
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS) inter_overflow_kernel(SearchParams P, const uint32_t *__restrict__ list,
                                                                 const uint32_t *__restrict__ count) {
  static_assert(THREADS >= 256, "one thread per position of a 16x16 window");
  depend();
  release_next();
  const int n = (int)__ldcg(count);
  if ((int)blockIdx.x >= n) return;  // the whole CTA, before its barriers
  __shared__ BlockTab s_tab;
  __shared__ uint8_t s_snap5[256], s_snap6[256];
  __shared__ int s_red[2 * (THREADS / 32)];
  __shared__ int s_sumsq;
  build_snap_tables(s_snap5, s_snap6);
  CtaReduce<THREADS> red{s_red, 0};
  for (int k = blockIdx.x; k < n; k += gridDim.x)
    cta_block_search<THREADS>(P, (int)__ldcg(list + k), s_tab, s_snap5, s_snap6, red, &s_sumsq);
}

}  // namespace mptc
