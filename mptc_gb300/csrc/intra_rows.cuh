// The intra search of a whole intra frame (IntraSearch,
// codec/dxt_image.cpp:652-713) for sa <= 8 as a pipeline over block rows.
#pragma once
#include <cstddef>
#include <cstdint>

#include "completion.cuh"

namespace mptc {

// ---- cluster helpers ---------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();  // the barrier wants whole warps
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of this CTA's shared variable p in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_map(const void *p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, uint64_t v) {
  asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}
__device__ __forceinline__ uint64_t ld_shared_relaxed(const uint64_t *p) {
  uint64_t v;
  asm volatile("ld.relaxed.cluster.shared::cta.u64 %0, [%1];"
               : "=l"(v)
               : "r"((uint32_t)__cvta_generic_to_shared(p))
               : "memory");
  return v;
}

// A cluster of CTAs takes a row of blocks at a time, rows in order from a
// counter; its CTAs take the row's groups of kRowGroup blocks in turn. A block
// needs the final index words of rows y-2sa+1 .. y-1 (columns x-sa .. x+sa-1)
// and of its sa left neighbours. The older ones are worked off ahead, by the
// kRowGroup worker warps of the group's CTA:
//  A. the distinct words of rows y-2sa+1 .. y-4 of the union of the group's
//     windows go into a hash table (the group's dictionary), with the union's
//     columns that hold each; worker k then evaluates those of block k's window
//     and takes the selection's statistics (selection.cuh) over its positions;
//  B. rows y-3 and y-2, one position per lane: looked up, new words evaluated;
//  C. the same for row y-1; the statistics reduced over the warp and left in
//     the block's mailbox.
// The last step is the row's only serial chain, kept in one warp per CTA:
//  D. the chain warp holds the last words in its lanes, looks all of the
//     block's left neighbours up at once, selects with one reduction, publishes
//     the block's word and passes on to the next block; after the group the
//     words go to the next group's CTA.
// The words that a neighbour can take, those of its window and its own stb
// word, are evaluated beforehand: the stb words of row y-1's and the left
// neighbours are entered as words without a position. A word that is not (it
// came from outside this window) is evaluated when it appears.
// Rows are decided in claim order by running clusters, so the waits always
// end; each is bounded like wait_done.
//
// Positions are numbered 16 * row + column in scan order (rows y, y-1, ..,
// columns x+sa-1 .. x-sa), which orders them as the reference's scan does.
// A final word is published as done_src(src, word): src is the block whose stb
// word it is, so that its refit weight sums are read (P.wdesc[src]) instead of
// summed again.
//
// Several frames at once are bound by the SMs that their CTAs hold: with two CTAs per
// SM (96 registers, a table of 768 buckets instead of 1024) the first frames of 8
// streams up to 2560x1440 and their 15 learned inter frames take 25.3 ms, with one 27.9.
//
// Bound by latency: the critical path of an intra frame is bw + sa * bh steps
// from a block to its right neighbour or to the row below, with one warp's chains of
// dependent instructions (about 5 cycles each) on them. So whatever can be known
// before the last neighbour is taken off that path, and a row's work is spread over
// four SMs. Clock stamps at 1080p and sa 8: a block takes the chain some 680 cycles,
// 320 of instructions, as many waiting for its mail (every fourth block) and 35 in
// row_decide (every 30th); a row takes 190 us and follows the one above by 5.3 us, so
// that 36 rows are in flight, about as many as there are clusters. A 1080p frame 1.43 to
// 1.52 ms, a 256x256 one 0.28 to 0.32, against 3.66 and 0.86 with one CTA per block polling
// global memory (intra_search_kernel). When it took 1.54 ms, clusters of 2, 3, 5 and
// 6 CTAs took 2.2, 1.77, 1.54 and 1.9, two sets of workers per CTA 1.8.
constexpr int kRowCluster = 4;  // CTAs per row
constexpr int kRowGroup = 8;    // blocks per group, worker warps per CTA
constexpr int kRowThreads = 32 * (kRowGroup + 1);
constexpr int kRowBack = 8;               // union columns to the left of the group's windows
constexpr int kRowCols = kRowGroup + 15 + kRowBack;  // union columns at sa = 8
constexpr int kRowOld = 12;               // rows y-4 .. y-15
// At most 12 * 31 words of step A, 55 without a position, 3 * 31 of rows y-3 ..
// y-1 and 15 left neighbours: the table never fills.
constexpr int kRowBuckets = 768;
constexpr int kRowAll = 128;  // up to so many words of step A are evaluated on every block
constexpr uint16_t kNoBucket = 0xFFFFu;
constexpr uint32_t kNoMatch = 0x100u;  // above every position
constexpr uint64_t kRowWord = 0x07FFFFFFFFFFFFFFull;  // a final word without its tag
static_assert(kRowCols <= 31, "union columns fit a mask; rounds of 32 hold a row's columns");

__device__ __forceinline__ uint64_t done_src(uint32_t src, uint32_t word) {
  return ((uint64_t)(src + 1u) << 32) | word;
}

struct __align__(16) RowDict {
  unsigned long long key[kRowBuckets];  // done_src of the word, 0: empty
  uint32_t cols[kRowBuckets];           // union columns holding it
  uint16_t list[kRowBuckets];           // the buckets in use by step A
  uint16_t at[kRowOld][32];             // the bucket of each position's word
  uint32_t count;
};
struct __align__(16) RowWork {
  BlockTab tab;
  uint32_t own;               // the block's own word,
  int orig, sumsq;            // its stb error and sum of squares
  uint32_t pad;
  uint2 ent[kRowBuckets];     // the bucket's word and its err_diff; the block's own word and 0 before that
  uint32_t eps[kRowBuckets];  // its endpoints
  uint16_t list[kRowBuckets];
};
// What the chain needs of a block, and its answer. The chain and the workers read
// each other's words while they are written, without a fence on the chain's path:
// every 64-bit half of a vector is written and read whole, is complete by itself and
// carries the group's tag in its top bits, so it does not matter in which order
// they are seen. The tables' entries are as complete (a word and its err_diff); the
// chain reads them behind the barrier that follows their reset (group_ready).
struct __align__(16) RowMail {
  uint64_t base;       // the word selected without the left neighbours, or the block's own
  uint32_t wins;       // (max(err_diff, 0) << 5 | lane) below which a left neighbour wins
  uint32_t pos;        // position of base (kNoMatch: not accepted), that of later << 16, tag
  uint64_t later;      // the word of the last row's err_diff < 0: an err_diff <= 0 gives way to it
  uint32_t own;
  uint32_t gives;      // 32 if there is such a word, else 0; tag
  uint64_t word;       // the chain's answer: the final word, for the blocks to its right;
  uint64_t answer;     // its index word and, above it, its position (kNoMatch: not accepted), for the worker
};
struct RowShared {
  RowDict dict;
  RowWork w[kRowGroup];
  RowMail mail[kRowGroup];
  uint64_t hist[8];  // the words before the CTA's next group, tagged with the group
  uint64_t row;
  uint8_t snap5[256], snap6[256];
};

static_assert(sizeof(RowDict) % 16 == 0 && offsetof(RowWork, ent) % 16 == 0 && offsetof(RowMail, later) % 16 == 0 &&
                  offsetof(RowMail, word) % 16 == 0,
              "vector accesses of the tables and the mail");

__device__ __forceinline__ uint32_t row_hash(uint32_t w) {
  return __umulhi(w * 2654435761u, (uint32_t)kRowBuckets);
}
__device__ __forceinline__ uint32_t row_after(uint32_t b) { return b + 1u < (uint32_t)kRowBuckets ? b + 1u : 0u; }
// The tag of group g's words (never 0 on the row's first lap).
__device__ __forceinline__ uint64_t row_tag(int g) { return (uint64_t)((g + 1) & 31) << 59; }
template <class T>
__device__ __forceinline__ T ld_volatile(const T *p) {
  return *reinterpret_cast<const volatile T *>(p);
}

// Two adjacent 64-bit words, each read or written whole: x, y and z, w.
__device__ __forceinline__ uint4 ld_shared_2x64(const void *p) {
  uint64_t a, b;
  asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];"
               : "=l"(a), "=l"(b)
               : "r"((uint32_t)__cvta_generic_to_shared(p))
               : "memory");
  return make_uint4((uint32_t)a, (uint32_t)(a >> 32), (uint32_t)b, (uint32_t)(b >> 32));
}
__device__ __forceinline__ void st_shared_2x64(void *p, uint4 v) {
  asm volatile("st.volatile.shared.v2.u64 [%0], {%1, %2};" ::"r"((uint32_t)__cvta_generic_to_shared(p)),
               "l"((uint64_t)v.y << 32 | v.x), "l"((uint64_t)v.w << 32 | v.z)
               : "memory");
}

// A bounded wait's clock, asked once per turn of a warp's waiting loop: true (in
// every lane) when it is over (~1 s, or another wait of the launch gave up).
struct WaitLimit {
  uint64_t t0 = 0;
  uint32_t it = 0;
  __device__ __forceinline__ bool warp_over(uint32_t *status) {
    return (++it & 31u) == 0u && __any_sync(kFull, check(status));
  }
  __device__ __forceinline__ bool check(uint32_t *status) {
    const uint64_t now = global_ns();
    if (t0 == 0) t0 = now;
    if (ld_acquire(status) & kDevTimeout) return true;
    if (now - t0 < 1000000000ull) return false;
    atomicOr(status, kDevTimeout);
    return true;
  }
};

// The bucket of the word of w, entered if it is not in the dictionary.
__device__ __forceinline__ uint32_t row_enter(RowDict &D, uint64_t w, bool &is_new) {
  uint32_t b = row_hash((uint32_t)w);
  for (int probe = 0; probe < kRowBuckets; ++probe) {
    const unsigned long long old = atomicCAS(&D.key[b], 0ull, (unsigned long long)w);
    is_new = old == 0ull;
    if (is_new || (uint32_t)old == (uint32_t)w) break;
    b = row_after(b);
  }
  return b;
}

// Whether block W has an err_diff for `word` (not its own), and which.
__device__ __forceinline__ bool row_find(const RowDict &D, const RowWork &W, uint32_t word, int &e) {
  uint32_t b = row_hash(word);
  for (int probe = 0; probe < kRowBuckets; ++probe) {
    const unsigned long long k = ld_volatile(&D.key[b]);
    if (k == 0ull) return false;
    if ((uint32_t)k == word) {
      const unsigned long long v = ld_volatile(reinterpret_cast<const unsigned long long *>(&W.ent[b]));
      e = (int)(uint32_t)(v >> 32);
      return (uint32_t)v == word;
    }
    b = row_after(b);
  }
  return false;
}

// The selection's statistics (selection.cuh) over some positions: the first
// err_diff <= 0; the first err_diff < 0 of the last row holding one (row << 8 |
// 255 - position); the first minimum ((err_diff + 65536) << 8 | position).
struct RowSel {
  int le0 = 0x7fffffff, neg = -1;
  uint32_t mn = 0xFFFFFFFFu;
  __device__ __forceinline__ void add(int e, int pos) {
    if (e == kInvalid) return;
    if (e <= 0) le0 = min(le0, pos);
    if (e < 0) neg = max(neg, ((pos >> 4) << 8) | (255 - pos));
    mn = min(mn, ((uint32_t)(e + 65536) << 8) | (uint32_t)pos);
  }
  __device__ __forceinline__ void reduce() {
    le0 = __reduce_min_sync(kFull, le0);
    neg = __reduce_max_sync(kFull, neg);
    mn = __reduce_min_sync(kFull, mn);
  }
};

// Evaluates the word of w on a block and keeps the result in bucket b.
__device__ __forceinline__ int row_eval(const RowShared &S, RowWork &W, const SearchParams &P, const PixelGroups &pg,
                                        uint64_t w, uint32_t b, uint32_t own, int orig, int sumsq) {
  const float4 d = __ldg(P.wdesc + ((uint32_t)(w >> 32) - 1u));
  const WeightSums ws{d.x, d.y, d.z, d.w};
  uint32_t eps = 0;
  int refit = 0;
  const int e = eval_candidate(W.tab, pg, S.snap5, S.snap6, (uint32_t)w, ws, own, orig, sumsq, eps, refit);
  W.eps[b] = eps;
  *reinterpret_cast<volatile unsigned long long *>(&W.ent[b]) = ((unsigned long long)(uint32_t)e << 32) | (uint32_t)w;
  return e;
}

// Each lane's word w (0: none), looked up; those without a result are
// evaluated side by side (equal ones in each of their lanes).
__device__ __forceinline__ int row_value(const RowShared &S, RowDict &D, RowWork &W, const SearchParams &P,
                                         const PixelGroups &pg, uint64_t w, uint32_t own, int orig, int sumsq) {
  int e = 0;
  const bool miss = w != 0ull && (uint32_t)w != own && !row_find(D, W, (uint32_t)w, e);
  if (__any_sync(kFull, miss)) {
    if (miss) {
      bool is_new;
      const uint32_t b = row_enter(D, w, is_new);
      e = row_eval(S, W, P, pg, w, b, own, orig, sumsq);
    }
    __syncwarp();
  }
  return w == 0ull ? kInvalid : (uint32_t)w == own ? 0 : e;
}

// All worker warps of the CTA.
__device__ __forceinline__ void worker_barrier() {
  __syncwarp();  // the barrier wants whole warps
  asm volatile("bar.sync 1, %0;" ::"n"(32 * kRowGroup) : "memory");
}

// The group's tables are reset and its blocks staged: worker 0 behind a barrier of all
// workers, to the chain. A worker gets there whether or not its waits gave up, and the
// chain asks once for each of its groups.
__device__ __forceinline__ void group_ready() {
  __syncwarp();
  asm volatile("bar.arrive 2, 64;" ::: "memory");
}
__device__ __forceinline__ void await_group() {
  __syncwarp();
  asm volatile("bar.sync 2, 64;" ::: "memory");
}

// One group's block by worker k (see above): steps A to C, then the answer
// written out.
__device__ __forceinline__ void row_worker(RowShared &S, const SearchParams &P, int k, int g, int by, int lane) {
  RowDict &D = S.dict;
  RowWork &W = S.w[k];
  RowMail &M = S.mail[k];
  const int sa = P.sa, w2 = 2 * sa, bw = P.bw;
  const int x0 = g * kRowGroup, bx = x0 + k, idx = by * bw + bx;
  const bool block = bx < bw;  // the row's last group may be short
  const unsigned lt_mask = (1u << lane) - 1u;
  WaitLimit limit;
  bool dead = false;  // a wait gave up: the frame is invalid, nothing waits any more
  uint64_t stb = 0;
  int orig = 0, sumsq = 0;
  if (block) {
    stb = __ldg(P.stb + idx);
    orig = __ldg(P.orig_err + idx);
    sumsq = stage_block(W.tab, P.rgb, P.width, bx, by, lane);
    const uint32_t own = (uint32_t)(stb >> 32);
    if (lane == 0) {
      W.own = own;
      W.orig = orig;
      W.sumsq = sumsq;
    }
    for (int b = lane; b < kRowBuckets / 2; b += 32)
      reinterpret_cast<uint4 *>(W.ent)[b] = make_uint4(own, 0u, own, 0u);
  }
  const uint32_t own = (uint32_t)(stb >> 32);
  // A. the dictionary, by all workers
  worker_barrier();  // the previous group is done
  {
    const int t = 32 * k + lane;
    for (int i = t; i < kRowBuckets / 2; i += 32 * kRowGroup)
      reinterpret_cast<ulonglong2 *>(D.key)[i] = make_ulonglong2(0ull, 0ull);
    for (int i = t; i < kRowBuckets / 4; i += 32 * kRowGroup)
      reinterpret_cast<uint4 *>(D.cols)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (t == 0) D.count = 0;
  }
  worker_barrier();
  if (k == 0) group_ready();
  // rounds 0-11: a row of the union each, y-4 .. y-15; 12: the stb words of
  // row y-1; 13: those of the left neighbours in row y and of the group itself
  const int u0 = x0 - sa - kRowBack, nu = 2 * sa + kRowGroup - 1 + kRowBack;  // the union's columns
#pragma unroll 1
  for (int q = k; q < kRowOld + 2; q += kRowGroup) {
    const int i = u0 + lane, j = q < kRowOld ? by - 4 - q : q == kRowOld ? by - 1 : by;
    const bool on = lane < nu && i >= 0 && i < bw && j >= 0 &&
                    (q < kRowOld ? 4 + q < w2 : q == kRowOld || i < x0 + kRowGroup);
    uint64_t w = 0;
    if (q < kRowOld) {
      const uint64_t *at = P.done + (on ? (size_t)j * bw + i : 0);
      for (;;) {
        if (on && w == 0ull) w = ld_relaxed(at);
        if (!__any_sync(kFull, on && w == 0ull) || dead) break;
        __nanosleep(40);
        dead = limit.warp_over(P.status);
      }
    } else if (on) {
      const uint32_t src = (uint32_t)(j * bw + i);
      w = done_src(src, (uint32_t)(__ldg(P.stb + src) >> 32));
    }
    uint32_t b = kNoBucket;
    bool is_new = false;
    if (w != 0ull) {
      b = row_enter(D, w, is_new);
      atomicOr(&D.cols[b], 1u << lane);
    }
    if (q < kRowOld) D.at[q][lane] = (uint16_t)b;
    const unsigned newm = __ballot_sync(kFull, is_new);
    int s = 0;
    if (lane == 0 && newm) s = (int)atomicAdd(&D.count, (uint32_t)__popc(newm));
    s = __shfl_sync(kFull, s, 0) + __popc(newm & lt_mask);
    if (is_new) D.list[s] = (uint16_t)b;
  }
  worker_barrier();
  if (!block) return;
  const PixelGroups pg = load_groups(W.tab);
  {
    // the block's words
    const int n = (int)D.count;
    const uint32_t win = n <= kRowAll ? ~0u : ((1u << w2) - 1u) << (k + kRowBack);
    int nl = 0;
    for (int s0 = 0; s0 < n; s0 += 32) {
      const int s = s0 + lane;
      uint32_t b = 0;
      bool take = false;
      if (s < n) {
        b = D.list[s];
        take = (D.cols[b] & win) != 0u && (uint32_t)D.key[b] != own;
      }
      const unsigned tm = __ballot_sync(kFull, take);
      if (take) W.list[nl + __popc(tm & lt_mask)] = (uint16_t)b;
      nl += __popc(tm);
    }
    __syncwarp();
    for (int s = lane; s < nl; s += 32) {
      const uint32_t b = W.list[s];
      row_eval(S, W, P, pg, D.key[b], b, own, orig, sumsq);
    }
    __syncwarp();
  }
  const int cc = lane & 15, i1 = bx + sa - 1 - cc;
  const bool col_ok = cc < w2 && i1 >= 0 && i1 < bw;
  RowSel sel;
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    const int r = 4 + 2 * c + (lane >> 4);
    if (col_ok && r < w2 && by >= r) {
      const uint32_t b = D.at[r - 4][kRowBack + k + w2 - 1 - cc];
      if (b != kNoBucket) sel.add((int)W.ent[b].y, 64 + 32 * c + lane);
    }
  }
  // B. rows y-2 (lanes 0-15) and y-3
  uint64_t w23 = 0;
  if (w2 > 2) {
    const int r = 2 + (lane >> 4);
    const bool on = col_ok && r < w2 && by >= r;
    for (;;) {
      if (on && w23 == 0ull) w23 = ld_relaxed(P.done + (size_t)(by - r) * bw + i1);
      if (!__any_sync(kFull, on && w23 == 0ull) || dead) break;
      __nanosleep(20);
      dead = limit.warp_over(P.status);
    }
    sel.add(row_value(S, D, W, P, pg, w23, own, orig, sumsq), 32 + lane);
    // the left neighbours' windows reach further: their words are evaluated
    // too, but are no candidates
    const int i2 = bx - sa - 1 - (lane & 7), r2 = 2 + (lane >> 3);
    uint64_t w = 0;
    if (lane < 16 && i2 >= 0 && r2 < w2 && by >= r2) w = ld_relaxed(P.done + (size_t)(by - r2) * bw + i2);
    row_value(S, D, W, P, pg, w, own, orig, sumsq);
  }
  // the statistics of rows y-2 and older, and their words
  sel.reduce();
  const uint64_t self = done_src((uint32_t)idx, own);
  auto word_at = [&](int pos) {  // pos >= 32, the same in every lane
    const uint64_t a = __shfl_sync(kFull, w23, pos & 31);
    if (pos < 64) return a;
    const uint32_t bk = D.at[(pos >> 4) - 4][kRowBack + k + w2 - 1 - (pos & 15)];
    return bk == kNoBucket ? self : (uint64_t)D.key[bk];
  };
  const uint64_t le0_w = sel.le0 != 0x7fffffff ? word_at(sel.le0) : self;
  const uint64_t neg_w = sel.neg >= 0 ? word_at(255 - (sel.neg & 255)) : self;
  const uint64_t mn_w = sel.mn != 0xFFFFFFFFu ? word_at((int)(sel.mn & 255u)) : self;
  // C. row y-1
  uint64_t w1 = 0;
  RowSel c;
  {
    // lanes 16 .. 23: further columns, as above
    const int i = lane < 16 ? i1 : bx - sa - 1 - (lane & 7);
    const bool on = (lane < 16 ? col_ok : lane < 24 && i >= 0) && by >= 1;
    for (;;) {
      if (on && w1 == 0ull) w1 = ld_relaxed(P.done + (size_t)(by - 1) * bw + i);
      if (!__any_sync(kFull, on && w1 == 0ull) || dead) break;
      dead = limit.warp_over(P.status);
    }
    const int e = row_value(S, D, W, P, pg, w1, own, orig, sumsq);
    if (lane < 16) c.add(e, 16 + lane);
  }
  c.reduce();
  // the reference's selection without the left neighbours (row y-1 comes before
  // the older rows); a negative threshold accepts nothing
  const int thr = P.thr;
  const bool le0 = min(c.le0, sel.le0) != 0x7fffffff;
  const int neg = max(c.neg, sel.neg);  // an older row's, if it holds one
  const uint32_t mn = min(c.mn, sel.mn);
  const int min_e = mn != 0xFFFFFFFFu ? (int)(mn >> 8) - 65536 : kInvalid;
  const int first = min(c.le0, sel.le0), later_pos = neg >= 0 ? 255 - (neg & 255) : 0;
  const uint64_t c_later = __shfl_sync(kFull, w1, later_pos & 15);
  const uint64_t later = sel.neg >= 0 ? neg_w : c_later;
  int pos = -1;
  uint64_t base = self;
  {
    const int p = le0 ? first : (int)(mn & 255u);
    const uint64_t c_base = __shfl_sync(kFull, w1, p & 15);
    const bool ok = thr >= 0 && (le0 || min_e <= thr);
    if (ok) {
      pos = p;
      base = p < 32 ? c_base : le0 ? le0_w : mn_w;
      if (le0 && (neg >> 8) > (first >> 4)) {
        pos = later_pos;
        base = later;
      }
    }
  }
  const uint64_t tag = row_tag(g);
  if (lane == 0) {
    __threadfence_block();
    const uint64_t bt = base | tag;
    const uint32_t hi = (uint32_t)(tag >> 32);
    // err_diffs are at most 65025
    const uint32_t wins = thr < 0 ? 0u : (uint32_t)(min(le0 ? 0 : min_e, min(thr, 65535)) + 1) << 5;
    st_shared_2x64(&M.later, make_uint4((uint32_t)later, (uint32_t)(later >> 32) | hi, own,
                                        (neg >= 0 && thr >= 0 ? 32u : 0u) | hi));
    st_shared_2x64(&M.base, make_uint4((uint32_t)bt, (uint32_t)(bt >> 32), wins,
                                     (pos < 0 ? kNoMatch : (uint32_t)pos) | ((uint32_t)later_pos << 16) | hi));
  }
  // Until the chain answers, the left neighbours' words are evaluated as they
  // appear: lane d - 1 watches the neighbour at distance d, in its mail or,
  // before the group, among the words handed over.
  uint64_t ans = 0;
  {
    bool open = lane < sa && lane > 0 && bx > lane;
    const uint64_t *src = lane < k ? &S.mail[k - 1 - lane].word : S.hist + ((lane - k) & 7);
    const uint32_t hi = (uint32_t)(tag >> 32);
    for (;;) {
      uint64_t l = 0;
      if (open) {
        l = ld_volatile(src);
        if (((uint32_t)(l >> 32) ^ hi) >> 27) l = 0;
      }
      ans = ld_volatile(&M.answer);
      if (__any_sync(kFull, l != 0ull)) {
        if (l != 0ull) open = false;
        row_value(S, D, W, P, pg, l & kRowWord, own, orig, sumsq);
      }
      if (!__any_sync(kFull, (((uint32_t)(ans >> 32) ^ hi) >> 27) != 0u) || dead) break;
      __nanosleep(40);
      dead = limit.warp_over(P.status);
    }
  }
  __threadfence_block();
  if (lane == 0) {
    const uint32_t p = (uint32_t)(ans >> 32) & 0x1FFu, word = (uint32_t)ans;
    uint64_t blk = stb;
    if (p != kNoMatch && word != own) {
      uint32_t b = row_hash(word);
      for (int probe = 0; probe < kRowBuckets && (uint32_t)ld_volatile(&D.key[b]) != word; ++probe)
        b = row_after(b);
      blk = (uint64_t)ld_volatile(&W.eps[b]) | ((uint64_t)word << 32);
    }
    P.final_blk[idx] = blk;
    P.motion[idx] = p != kNoMatch ? (uint16_t)((w2 - 1 - (p & 15)) | ((w2 - 1 - (p >> 4)) << 8)) : (uint16_t)0xFFFFu;
  }
  __syncwarp();
}

// The chain's slow path for a block with mail (ma, mb): decides it from its left
// neighbours' words (lane d - 1: distance d; 0: none), searching the table to the
// end and evaluating those without a result. Returns the block's word and
// position in every lane.
struct RowAnswer {
  uint64_t word;
  uint32_t pos;
};
__device__ __noinline__ RowAnswer row_decide(RowShared &S, const SearchParams &P, int k, int nb, uint64_t h,
                                             uint4 ma, uint4 mb, int lane) {
  RowDict &D = S.dict;
  RowWork &W = S.w[k];
  if (lane >= P.sa) h = 0;
  // a word without a result is evaluated on this block and, lane by lane, on the
  // group's blocks after it
  int e = 0;
  const bool known = h == 0ull || (uint32_t)h == mb.z || row_find(D, W, (uint32_t)h, e);
  for (unsigned open = __ballot_sync(kFull, !known); open; open &= open - 1u) {
    const int l = __ffs(open) - 1;
    const uint64_t w = __shfl_sync(kFull, h, l);
    int v = 0;
    if (k + lane < nb) {
      RowWork &Wl = S.w[k + lane];
      if ((uint32_t)w != ld_volatile(&Wl.own) && !row_find(D, Wl, (uint32_t)w, v)) {
        bool is_new;
        const uint32_t b = row_enter(D, w, is_new);
        v = row_eval(S, Wl, P, load_groups(Wl.tab), w, b, ld_volatile(&Wl.own), ld_volatile(&Wl.orig),
                     ld_volatile(&Wl.sumsq));
      }
    }
    __syncwarp();
    __threadfence_block();  // before lane 0's answer, behind which the workers read
    v = __shfl_sync(kFull, v, 0);
    if (lane == l) e = v;
  }
  __syncwarp();
  if (h == 0ull) e = kInvalid;
  if ((uint32_t)h == mb.z && h != 0ull) e = 0;
  const uint32_t m = __reduce_min_sync(kFull, e != kInvalid ? ((uint32_t)max(e, 0) << 5) | (uint32_t)lane : 0xFFFFFFFFu);
  RowAnswer r;
  r.word = __shfl_sync(kFull, h, (int)(m & 31u));
  r.pos = (uint32_t)P.sa + (m & 31u);
  if (m >= ma.z) {
    r.word = (((uint64_t)ma.y << 32) | ma.x) & kRowWord;
    r.pos = ma.w & 0x1FFu;
  }
  if (m < (mb.w & 32u)) {
    r.word = (((uint64_t)mb.y << 32) | mb.x) & kRowWord;
    r.pos = (ma.w >> 16) & 255u;
  }
  return r;
}

// PER_SM: CTAs that an SM holds at once. A frame by itself is fastest with one (two
// of its CTAs on an SM slow the chain: 1.75 ms against 1.52 at 1080p), unless it is wide;
// wide frames and frames beside others' take half the registers and share the SMs
// (launch_intra_frame has the rule).
template <int PER_SM>
__global__ void __launch_bounds__(kRowThreads, PER_SM) intra_rows_kernel(SearchParams P) {
  extern __shared__ __align__(16) uint8_t row_smem[];
  RowShared &S = *reinterpret_cast<RowShared *>(row_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rank = cluster_rank(), ncta = cluster_size();
  build_snap_tables(S.snap5, S.snap6);
  depend();
  const int sa = P.sa, bw = P.bw, groups = (bw + kRowGroup - 1) / kRowGroup;
  const uint32_t next_hist = cluster_map(S.hist, (rank + 1u) % ncta);
  for (;;) {
    cluster_sync();  // the previous row is decided
    if (tid < kRowGroup) S.mail[tid] = RowMail{};
    if (tid < 8) S.hist[tid] = 0;
    if (rank == 0 && tid == 0) {
      const uint32_t y = atomicAdd(P.work, 1u);
      for (uint32_t r = 0; r < ncta; ++r) st_cluster(cluster_map(&S.row, r), y);
    }
    __syncwarp();
    cluster_sync();
    const int by = (int)ld_shared_relaxed(&S.row);
    if (by >= P.bh) break;
    if (warp < kRowGroup) {
#pragma unroll 1
      for (int g = (int)rank; g < groups; g += (int)ncta) row_worker(S, P, warp, g, by, lane);
    } else {
      // D. the chain: lane d - 1 holds the word of the left neighbour at distance d
      bool dead = false;
      uint64_t h = 0;
#pragma unroll 1
      for (int g = (int)rank; g < groups; g += (int)ncta) {
        await_group();
        if (g > 0 && ncta > 1) {
          const uint32_t tag = (uint32_t)(row_tag(g) >> 59);
          WaitLimit limit;
          uint64_t t = 0;
          while (!dead) {
            if (lane < 8) t = ld_shared_relaxed(S.hist + lane);
            if (__all_sync(kFull, lane >= 8 || (uint32_t)(t >> 59) == tag)) break;
            dead = limit.warp_over(P.status);
          }
          h = dead ? 0ull : t & kRowWord;
        }
        // lane d - 1 looks the left neighbour at distance d up in the block's
        // table (nearly always in its first two buckets) and one reduction
        // finds the best: the smallest err_diff, those <= 0 alike, then the
        // nearest, which is the first in scan order. The lanes of one load need not see the same
        // store, so they decide together.
        const uint32_t tag = (uint32_t)(row_tag(g) >> 32);
        uint32_t hlo = (uint32_t)h, hhi = (uint32_t)(h >> 32);  // h in halves
        const int nb = min(kRowGroup, bw - g * kRowGroup);
        const RowWork *W = S.w;
        RowMail *M = S.mail;
        uint64_t *done = P.done + (size_t)by * bw + g * kRowGroup;
#pragma unroll 1
        for (int k = 0; k < nb && !dead; ++k, ++W, ++M, ++done) {
          const uint32_t lo = hlo, hi = hhi, hb = row_hash(lo);
          const bool on = hi != 0u && lane < sa;
          uint4 ma, mb;
          uint32_t m;
          bool slow;
          WaitLimit limit;
          for (;;) {  // until the block's mail is there
            ma = ld_shared_2x64(&M->base);
            mb = ld_shared_2x64(&M->later);
            unsigned long long v = ld_volatile(reinterpret_cast<const unsigned long long *>(&W->ent[hb]));
            const unsigned long long v2 = ld_volatile(
                reinterpret_cast<const unsigned long long *>(&W->ent[row_after(hb)]));
            if ((uint32_t)v != lo) v = v2;
            const bool wait = ((tag ^ ma.y) | (tag ^ ma.w) | (tag ^ mb.y) | (tag ^ mb.w)) >= 1u << 27;
            m = __reduce_min_sync(kFull, on ? ((uint32_t)max((int)(v >> 32), 0) << 5) | (uint32_t)lane : 0xFFFFFFFFu);
            slow = __any_sync(kFull, wait || (on && (uint32_t)v != lo));
            if (!slow || !__any_sync(kFull, wait)) break;
            dead = limit.warp_over(P.status);
            if (dead) break;
          }
          if (dead) break;  // the workers' waits give up too
          // the words move one lane up; lane 0 takes the block's (whi and pos with the tag)
          const int from = lane == 0 ? (int)(m & 31u) : lane - 1;
          const uint32_t nlo = __shfl_sync(kFull, lo, from), nhi = __shfl_sync(kFull, hi, from);
          uint32_t wlo = nlo, whi = nhi | tag;
          uint32_t pos = tag + (uint32_t)sa + (m & 31u);
          if (m >= ma.z) {
            wlo = ma.x, whi = ma.y;
            pos = ma.w & 0xF80001FFu;
          }
          if (m < (mb.w & 32u)) {
            wlo = mb.x, whi = mb.y;
            pos = tag | (ma.w >> 16 & 255u);
          }
          if (slow) {
            const RowAnswer r = row_decide(S, P, k, nb, (uint64_t)hhi << 32 | hlo, ma, mb, lane);
            wlo = (uint32_t)r.word, whi = (uint32_t)(r.word >> 32) | tag;
            pos = r.pos | tag;
          }
          const uint32_t wsrc = whi & 0x07FFFFFFu;
          hlo = lane == 0 ? wlo : nlo;
          hhi = lane == 0 ? wsrc : nhi;
          if (lane == 0) {
            st_relaxed(done, (uint64_t)wsrc << 32 | wlo);
            st_shared_2x64(&M->word, make_uint4(wlo, whi, wlo, pos));
          }
          __syncwarp();
        }
        h = (uint64_t)hhi << 32 | hlo;
        if (lane < 8 && g + 1 < groups && ncta > 1)
          st_cluster(next_hist + 8u * (uint32_t)lane, h | row_tag(g + 1));
      }
    }
    __syncwarp();
  }
}

}  // namespace mptc
