// Training and embedding kernels of the learned candidate proposal (see
// learned_common.cuh for the model): tensor-core GEMM with transposes and
// fused bias/ReLU, feature builders, sampled softmax cross-entropy, AdamW.
#pragma once
#include "completion.cuh"
#include "learned_common.cuh"
#include "tc_sm100.cuh"

namespace mptc {

// C[M x N] = op(A)[M x K] * op(B)[K x N], then the epilogue GemmEpi, on the
// fifth-generation tensor cores: BF16 operands, FP32 accumulators in TMEM.
// TA: A is stored K x M (row-major, lda), else M x K; TB: B is stored N x K,
// else K x N. Split K (gridDim.z > 1): slice z writes its partial product to
// C + z * M * ldc and nothing else; the caller sums the slices in order.
//
// Tiles of 128 x BN (one TMEM lane per row), K in steps of 64 through up to two
// shared-memory stages in the 128-byte-swizzled K-major layout (rows of 64 K
// values). Each thread holds its share of the next step's operand tiles in
// registers while the tensor cores work on the current one: an operand whose
// K run is contiguous in memory (A not transposed, B transposed) moves as
// 16-byte vectors, the other is read 8 rows (or columns) at a time along its
// contiguous dimension and goes into the tile's rows through a register
// transpose. Thread 0 issues 4 tcgen05.mma (K = 16 each) per step and commits
// them to the stage's mbarrier; a stage is refilled once the MMAs that read it
// have completed. In the epilogue each warp moves its 32 accumulator rows
// through its own shared memory 64 columns at a time, so that a lane owns two
// adjacent columns and every warp store covers a whole row segment.
//
// What bounds these products is latency, not their arithmetic: one to five
// steps between the loads and the epilogue of a CTA, hidden only by the other
// CTAs of the SM. Hence one stage where K needs no second (36 KB, four CTAs an
// SM instead of three), BN = 64 where N is 64 or 128-wide tiles would leave SMs
// idle, and no block barrier in the epilogue. The products of 131072 candidate
// rows took 35 (32 x 128), 34 (128 x 64) and 54 us (dx, 64 x 128) with three CTAs an SM
// and block-wide staging of 32 columns, now 25, 25 and 37.
constexpr int kTcBM = 128, kTcBK = 64;
template <int BN>
__host__ __device__ constexpr int tc_stage() { return (kTcBM + BN) * 128; }  // bytes: A and B tiles
constexpr int kTcPitch = 66;                                // floats per staged row of 64 columns
constexpr int kTcEpi = (kTcBM * kTcPitch + 4 * 128) * 4;    // the warps' staged rows, their column sums
// Dynamic shared memory for a slice of K of `steps` steps: its stages or the
// epilogue's staging, and alignment slack.
template <int BN>
constexpr int tc_smem(int steps) {
  return (tc_stage<BN>() * (steps < 2 ? 1 : 2) > kTcEpi ? tc_stage<BN>() * (steps < 2 ? 1 : 2) : kTcEpi) + 1024;
}
// K steps of a slice when K is split over z slices.
__host__ __device__ inline int tc_steps(int K, int z) { return ((K + z - 1) / z + kTcBK - 1) / kTcBK; }

// Epilogue of gemm_tc_kernel, applied in this order to each output x:
// + bias[n]; ReLU; x = 0 where mask[m * ldc + n] <= 0 (ReLU backward); then
// C (fp32) and/or Cb (bf16) receive x, and colpart[blockIdx.y * ldc + n] the
// sum of x over the tile's rows (rows in a fixed order: the same bits every
// run). Null pointers skip their step. N is even; C, Cb and mask are aligned to
// two elements.
struct GemmEpi {
  float *C;
  __nv_bfloat16 *Cb;
  int ldc;
  const float *bias;
  int relu;
  const __nv_bfloat16 *mask;
  float *colpart;
};

// Eight consecutive bf16 at p, of which the first `valid` exist (zeros after):
// one 16-byte load when all eight exist and p is 16-byte aligned.
__device__ __forceinline__ uint4 load8_bf16(const __nv_bfloat16 *p, int valid) {
  if (valid >= 8 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) return *reinterpret_cast<const uint4 *>(p);
  uint16_t h[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) h[j] = j < valid ? reinterpret_cast<const uint16_t *>(p)[j] : (uint16_t)0;
  return make_uint4(h[0] | ((uint32_t)h[1] << 16), h[2] | ((uint32_t)h[3] << 16), h[4] | ((uint32_t)h[5] << 16),
                    h[6] | ((uint32_t)h[7] << 16));
}

// One ROWS x 64 operand tile (rows row0 .. row0 + ROWS - 1 of nrows, K values
// k0 .. k0 + 63 below kend; zeros outside) in this thread's registers.
// KMAJOR: src[row][k], stride ld: register i is K values 8 (t % 8) .. of row
// t / 8 + 16 i. Otherwise src[k][row]: register i is rows 8 (t / 8) .. of K
// value 8 (t % 8) + i.
template <bool KMAJOR, int ROWS>
__device__ __forceinline__ void load_tile(uint4 (&r)[8], const __nv_bfloat16 *__restrict__ src, int ld, int row0,
                                          int nrows, int k0, int kend, int tid) {
  const int kb = tid & 7;
#pragma unroll
  for (int i = 0; i < (KMAJOR ? ROWS / 16 : 8); ++i) {
    r[i] = make_uint4(0u, 0u, 0u, 0u);
    if (KMAJOR) {
      const int row = row0 + (tid >> 3) + 16 * i, k = k0 + 8 * kb;
      if (row < nrows && k < kend) r[i] = load8_bf16(src + (size_t)row * ld + k, kend - k);
    } else {
      const int row = row0 + 8 * (tid >> 3), k = k0 + 8 * kb + i;
      if (8 * (tid >> 3) < ROWS && row < nrows && k < kend)
        r[i] = load8_bf16(src + (size_t)k * ld + row, nrows - row);
    }
  }
}

// Stores the registers of load_tile<KMAJOR> into the swizzled tile. The
// transposed case builds row r + j's 8 K values from element j of the 8
// registers: each output word is one byte permutation of two input words.
template <bool KMAJOR, int ROWS>
__device__ __forceinline__ void store_tile(uint8_t *tile, const uint4 (&r)[8], int tid) {
  const uint32_t kb = tid & 7;
  if (KMAJOR) {
#pragma unroll
    for (int i = 0; i < ROWS / 16; ++i)
      *reinterpret_cast<uint4 *>(tile + tc::sw128_offset((uint32_t)((tid >> 3) + 16 * i), kb)) = r[i];
  } else if (8 * (tid >> 3) < ROWS) {
    const uint32_t w[8][4] = {{r[0].x, r[0].y, r[0].z, r[0].w}, {r[1].x, r[1].y, r[1].z, r[1].w},
                              {r[2].x, r[2].y, r[2].z, r[2].w}, {r[3].x, r[3].y, r[3].z, r[3].w},
                              {r[4].x, r[4].y, r[4].z, r[4].w}, {r[5].x, r[5].y, r[5].z, r[5].w},
                              {r[6].x, r[6].y, r[6].z, r[6].w}, {r[7].x, r[7].y, r[7].z, r[7].w}};
    const uint32_t row = 8u * (uint32_t)(tid >> 3);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t sel = (j & 1) ? 0x7632u : 0x5410u;
      const uint4 o = make_uint4(__byte_perm(w[0][j >> 1], w[1][j >> 1], sel),
                                 __byte_perm(w[2][j >> 1], w[3][j >> 1], sel),
                                 __byte_perm(w[4][j >> 1], w[5][j >> 1], sel),
                                 __byte_perm(w[6][j >> 1], w[7][j >> 1], sel));
      *reinterpret_cast<uint4 *>(tile + tc::sw128_offset(row + (uint32_t)j, kb)) = o;
    }
  }
}

template <bool TA, bool TB, int BN>
__global__ void __launch_bounds__(128, TA && BN == 128 ? 3 : 4)
    gemm_tc_kernel(const __nv_bfloat16 *__restrict__ A, int lda, const __nv_bfloat16 *__restrict__ B, int ldb,
                   GemmEpi ep, int M, int N, int K, uint32_t *__restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = tc::align_1024(smem_raw);
  __shared__ uint64_t bar[2];
  __shared__ uint32_t tslot;
  __shared__ volatile uint32_t abort_flag, drain_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * kTcBM, n0 = blockIdx.x * BN;
  depend();
  release_next();
  // split K (blockIdx.z): this slice's K range, in whole steps
  const int kstep = tc_steps(K, gridDim.z) * kTcBK;
  const int kbeg = blockIdx.z * kstep, kend = min(K, kbeg + kstep);
  const int steps = kend > kbeg ? (kend - kbeg + kTcBK - 1) / kTcBK : 0;
  uint4 ra[8], rb[8];
  if (steps > 0) {
    load_tile<!TA, kTcBM>(ra, A, lda, m0, M, kbeg, kend, tid);
    load_tile<TB, BN>(rb, B, ldb, n0, N, kbeg, kend, tid);
  }
  if (tid == 0) {
    tc::mbar_init(&bar[0], 1);
    tc::mbar_init(&bar[1], 1);
    abort_flag = 0;
    drain_flag = 0;
    tc::mbar_fence_init();
  }
  __syncwarp();
  if (warp == 0) tc::tmem_alloc(&tslot, BN);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = tslot;
  const uint32_t idesc = tc::idesc_bf16(kTcBM, BN);
  // A wait that gives up sets abort_flag: the remaining waits return at once,
  // the steps still run (uniform control flow) and the results are reported
  // invalid through *status.
  for (int s = 0; s < steps; ++s) {
    const int st = s & 1;
    uint8_t *sA = smem + st * tc_stage<BN>(), *sB = sA + kTcBM * 128;
    // the MMAs of step s - 2 read this stage
    if (s >= 2 && !tc::mbar_wait(&bar[st], (uint32_t)((s - 2) >> 1) & 1u, &abort_flag)) abort_flag = 1;
    store_tile<!TA, kTcBM>(sA, ra, tid);
    store_tile<TB, BN>(sB, rb, tid);
    tc::fence_async_smem();
    __syncthreads();
    if (tid == 0) {
      tc::tc_fence_after();
      const uint32_t a = tc::smem_addr(sA), b = tc::smem_addr(sB);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        tc::mma_bf16(tmem, tc::desc_sw128(a + 32 * k), tc::desc_sw128(b + 32 * k), idesc, (s > 0 || k > 0) ? 1u : 0u);
      tc::mma_commit(&bar[st]);
    }
    if (s + 1 < steps) {
      const int k0 = kbeg + (s + 1) * kTcBK;
      load_tile<!TA, kTcBM>(ra, A, lda, m0, M, k0, kend, tid);
      load_tile<TB, BN>(rb, B, ldb, n0, N, k0, kend, tid);
    }
  }
  // every MMA has completed once the last step's commit has arrived
  const uint32_t last_parity = (uint32_t)((steps - 1) >> 1) & 1u;
  if (steps > 0 && !tc::mbar_wait(&bar[(steps - 1) & 1], last_parity, &abort_flag)) abort_flag = 1;
  tc::tc_fence_after();
  const bool failed = __syncthreads_or(abort_flag != 0) != 0;
  if (failed) {
    // let MMAs still in flight finish (bounded) before the TMEM is freed
    if (steps > 0) tc::mbar_wait(&bar[(steps - 1) & 1], last_parity, &drain_flag, 100000000ull);
    if (tid == 0 && status) atomicOr(status, 1u);
  } else {
    // epilogue: the warp's rows m0 + 32 warp .. + 31, lane = two columns
    float *stg = reinterpret_cast<float *>(smem) + warp * 32 * kTcPitch;
    float *csum = reinterpret_cast<float *>(smem) + kTcBM * kTcPitch;  // [4 warps][128]
    const uint32_t lane_base = tmem + ((uint32_t)(32 * warp) << 16);
    const int mw = m0 + 32 * warp, rows = min(32, M - mw);
    const bool split = gridDim.z > 1;
#pragma unroll 1
    for (int c0 = 0; c0 < BN && n0 + c0 < N; c0 += 64) {
      const int n = n0 + c0 + 2 * lane;
      // the mask's values are read before any store (a store through another
      // pointer could otherwise order each read after it)
      uint32_t mk[32];
      if (!TA && ep.mask) {
#pragma unroll
        for (int i = 0; i < 32; ++i)
          mk[i] = n < N && i < rows ? *reinterpret_cast<const uint32_t *>(ep.mask + (size_t)(mw + i) * ep.ldc + n) : 0u;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float v[32];
        tc::tmem_ld32(lane_base + (uint32_t)(c0 + 32 * h), v);
#pragma unroll
        for (int j = 0; j < 16; ++j)
          *reinterpret_cast<float2 *>(stg + lane * kTcPitch + 32 * h + 2 * j) =
              steps > 0 ? make_float2(v[2 * j], v[2 * j + 1]) : make_float2(0.f, 0.f);
      }
      __syncwarp();
      const float2 *mine = reinterpret_cast<const float2 *>(stg + 2 * lane);
      if (n < N && split) {
        float *Cz = ep.C + ((size_t)blockIdx.z * M + mw) * ep.ldc + n;
#pragma unroll 8
        for (int i = 0; i < 32; ++i)
          if (i < rows) *reinterpret_cast<float2 *>(Cz + (size_t)i * ep.ldc) = mine[i * (kTcPitch / 2)];
      } else if (n < N) {
        const float b0 = ep.bias ? ep.bias[n] : 0.f, b1 = ep.bias ? ep.bias[n + 1] : 0.f;
        float2 cs = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          if (i < rows) {
            const size_t o = (size_t)(mw + i) * ep.ldc + n;
            float2 x = mine[i * (kTcPitch / 2)];
            x.x += b0, x.y += b1;
            if (ep.relu) x.x = x.x > 0.f ? x.x : 0.f, x.y = x.y > 0.f ? x.y : 0.f;
            if (!TA && ep.mask) {
              if (!(__uint_as_float(mk[i] << 16) > 0.f)) x.x = 0.f;
              if (!(__uint_as_float(mk[i] & 0xFFFF0000u) > 0.f)) x.y = 0.f;
            }
            if (ep.C) *reinterpret_cast<float2 *>(ep.C + o) = x;
            if (ep.Cb) *reinterpret_cast<__nv_bfloat162 *>(ep.Cb + o) = __floats2bfloat162_rn(x.x, x.y);
            cs.x += x.x, cs.y += x.y;
          }
        }
        *reinterpret_cast<float2 *>(csum + 128 * warp + c0 + 2 * lane) = cs;
      }
      __syncwarp();
    }
    if (ep.colpart && !split) {
      __syncthreads();
      if (tid < BN && n0 + tid < N)
        ep.colpart[(size_t)blockIdx.y * ep.ldc + n0 + tid] =
            ((csum[tid] + csum[128 + tid]) + csum[256 + tid]) + csum[384 + tid];
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  if (warp == 0) tc::tmem_free(tmem, BN);
}

// Block features (block_feature_half) of blocks[r] (NULL: block r), n rows of
// kFeatPad bf16.
__global__ void block_features_kernel(const uint8_t *__restrict__ rgb, int width, int bw, const uint64_t *__restrict__ stb,
                                      const uint32_t *__restrict__ blocks, int n, __nv_bfloat16 *__restrict__ X) {
  depend();
  release_next();
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < 2 * n; e += gridDim.x * blockDim.x) {
    const int r = e >> 1, half = e & 1;
    const int idx = blocks ? (int)blocks[r] : r;
    const int by = idx / bw, bx = idx - by * bw;
    uint32_t f[16];
    block_feature_half(rgb, width, bx, by, stb[idx], half, f);
    uint4 *dst = reinterpret_cast<uint4 *>(X + (size_t)r * kFeatPad + 32 * half);
#pragma unroll
    for (int j = 0; j < 4; ++j) dst[j] = make_uint4(f[4 * j], f[4 * j + 1], f[4 * j + 2], f[4 * j + 3]);
  }
}

// Candidate features: the 32 bits of an index word as 0/1, 8 per thread and
// 16-byte store (one per thread took 10 us for 131072 words).
__global__ void cand_features_kernel(const uint32_t *__restrict__ words, int word_stride, int n,
                                     __nv_bfloat16 *__restrict__ X) {
  depend();
  release_next();
  const int total = n * (kCandIn / 8);
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
    const int r = e / (kCandIn / 8), c = e % (kCandIn / 8);
    const uint32_t bits = words[(size_t)r * word_stride] >> (8 * c);
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)  // 0x3F80 is one
      w[j] = ((bits >> (2 * j)) & 1u) * 0x3F80u | ((bits >> (2 * j + 1)) & 1u) * 0x3F800000u;
    reinterpret_cast<uint4 *>(X)[e] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

__global__ void bf16_to_f32_kernel(const __nv_bfloat16 *__restrict__ x, float *__restrict__ y, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = __bfloat162float(x[i]);
}

__global__ void to_bf16_kernel(const float *__restrict__ x, __nv_bfloat16 *__restrict__ y, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = __float2bfloat16(x[i]);
}

// The sums of a step's split reductions, all in one launch: for each job, out[i]
// = sum over slices k < slices of part[k * n + i], in a fixed order (the same
// bits every run): warp w of a CTA sums slices w, w + kSumWarps, ... for 32
// outputs of a job (lane = output) in four interleaved chains; the chains, then
// the warps, are added in order. Few outputs and up to 1024 slices: with 8 warps
// the chains of loads took 17 us; a launch per job, ten of the step's 27.
constexpr int kSumWarps = 32, kMaxSums = 10;
struct SumJob {
  const float *part;
  float *out;
  int slices, n;
  int end;  // CTAs of this job and those before it
};
struct SumJobs {
  SumJob job[kMaxSums];
  int n;
};
__global__ void __launch_bounds__(32 * kSumWarps) slice_sum_kernel(const __grid_constant__ SumJobs jobs) {
  __shared__ float red[kSumWarps][32];
  int q = 0;
  while (q + 1 < jobs.n && (int)blockIdx.x >= jobs.job[q].end) ++q;
  const SumJob &job = jobs.job[q];
  const float *__restrict__ part = job.part;
  const int slices = job.slices, n = job.n;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = (blockIdx.x - (q ? jobs.job[q - 1].end : 0)) * 32 + lane;
  float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
  if (i < n) {
    int k = warp;
#pragma unroll 2
    for (; k + 3 * kSumWarps < slices; k += 4 * kSumWarps) {
      a0 += part[(size_t)k * n + i];
      a1 += part[(size_t)(k + kSumWarps) * n + i];
      a2 += part[(size_t)(k + 2 * kSumWarps) * n + i];
      a3 += part[(size_t)(k + 3 * kSumWarps) * n + i];
    }
    for (; k < slices; k += kSumWarps) a0 += part[(size_t)k * n + i];
  }
  red[warp][lane] = (a0 + a1) + (a2 + a3);
  __syncthreads();
  if (warp == 0 && i < n) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kSumWarps; ++w) t += red[w][lane];
    job.out[i] = t;
  }
}

constexpr int kMaxCE = 64;  // candidates per block in one training example

// Sampled softmax cross-entropy: block b scores its C candidates (row b*C .. of
// G) against F[b]; candidate 0 is the accepted one. Adds the mean loss
// (atomic) and writes the bf16 gradients dF [B x 64] and dG [B*C x 64], and
// for the bias gradients the fp32 column sums of each CTA's rows of dF and
// dG: partF / partG [gridDim.x x 64] (fixed order: candidates, then warps).
// One warp per block, 8 blocks per CTA of 256 threads, lane = dims 2 lane and
// 2 lane + 1. Eight candidates at a time: their rows are loaded together and
// their eight dot products reduced together (9 shuffles instead of 40), which
// leaves candidate 8 k + q's score in lanes 4 q .. 4 q + 3, register k. One
// candidate at a time, with the scores in local memory, took 25 us for 4096
// blocks of 32 candidates.
__global__ void __launch_bounds__(256) softmax_ce_kernel(const float *__restrict__ F, const float *__restrict__ G,
                                                         int B, int C, __nv_bfloat16 *__restrict__ dF,
                                                         __nv_bfloat16 *__restrict__ dG, float *__restrict__ partF,
                                                         float *__restrict__ partG, float *__restrict__ loss) {
  __shared__ float colF[8][kEmb], colG[8][kEmb];
  depend();
  release_next();
  constexpr unsigned kAll = 0xffffffffu;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.x * 8 + w;
  float2 df = make_float2(0.f, 0.f), cg = make_float2(0.f, 0.f);
  if (b < B) {
    const float2 f = reinterpret_cast<const float2 *>(F + (size_t)b * kEmb)[lane];
    const float2 *g = reinterpret_cast<const float2 *>(G + (size_t)b * C * kEmb) + lane;
    float s[kMaxCE / 8];
    float mx = -1e30f;
#pragma unroll
    for (int k = 0; k < kMaxCE / 8; ++k) {
      s[k] = -1e30f;
      if (8 * k >= C) continue;
      float v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float2 x = 8 * k + q < C ? g[(8 * k + q) * (kEmb / 2)] : make_float2(0.f, 0.f);
        v[q] = f.x * x.x + f.y * x.y;
      }
#pragma unroll
      for (int h = 4; h > 0; h >>= 1) {
        const bool up = lane & (4 * h);
#pragma unroll
        for (int q = 0; q < h; ++q) {
          const float send = up ? v[q] : v[q + h], keep = up ? v[q + h] : v[q];
          v[q] = keep + __shfl_xor_sync(kAll, send, 4 * h);
        }
      }
      v[0] += __shfl_xor_sync(kAll, v[0], 2);
      v[0] += __shfl_xor_sync(kAll, v[0], 1);
      if (8 * k + (lane >> 2) < C) s[k] = v[0];
      mx = fmaxf(mx, s[k]);
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(kAll, mx, o));
    float z = 0.f;
#pragma unroll
    for (int k = 0; k < kMaxCE / 8; ++k)
      if (8 * k + (lane >> 2) < C) z += __expf(s[k] - mx);
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) z += __shfl_xor_sync(kAll, z, o);
    const float inv = 1.f / z;
    if (lane == 0) atomicAdd(loss, (mx + __logf(z) - s[0]) / B);
    __nv_bfloat162 *dg = reinterpret_cast<__nv_bfloat162 *>(dG + (size_t)b * C * kEmb) + lane;
#pragma unroll
    for (int k = 0; k < kMaxCE / 8; ++k) {
      if (8 * k >= C) continue;
      const float p = __expf(s[k] - mx) * inv;
      const float dsk = (p - (k == 0 && lane < 4 ? 1.f : 0.f)) / B;
      float2 x[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) x[q] = 8 * k + q < C ? g[(8 * k + q) * (kEmb / 2)] : make_float2(0.f, 0.f);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float ds = __shfl_sync(kAll, dsk, 4 * q);
        if (8 * k + q >= C) continue;
        df.x += ds * x[q].x;
        df.y += ds * x[q].y;
        const float d0 = ds * f.x, d1 = ds * f.y;
        dg[(8 * k + q) * (kEmb / 2)] = __floats2bfloat162_rn(d0, d1);
        cg.x += d0;
        cg.y += d1;
      }
    }
    reinterpret_cast<__nv_bfloat162 *>(dF + (size_t)b * kEmb)[lane] = __floats2bfloat162_rn(df.x, df.y);
  }
  reinterpret_cast<float2 *>(colF[w])[lane] = df;
  reinterpret_cast<float2 *>(colG[w])[lane] = cg;
  __syncthreads();
  const int t = threadIdx.x;
  if (t < 2 * kEmb) {
    const int c = t & (kEmb - 1);
    float(*col)[kEmb] = t < kEmb ? colF : colG;
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) acc += col[k][c];
    (t < kEmb ? partF : partG)[(size_t)blockIdx.x * kEmb + c] = acc;
  }
}

// AdamW on fp32 master weights, refreshing their bf16 copies.
__global__ void adamw_kernel(float *__restrict__ w, __nv_bfloat16 *__restrict__ wb, const float *__restrict__ grad,
                             float *__restrict__ m, float *__restrict__ v, int n, float lr, float b1, float b2,
                             float eps, float wd, float c1, float c2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float g = grad[i];
    const float mi = b1 * m[i] + (1.f - b1) * g, vi = b2 * v[i] + (1.f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float upd = (mi / c1) / (sqrtf(vi / c2) + eps) + wd * w[i];
    const float wi = w[i] - lr * upd;
    w[i] = wi;
    if (wb) wb[i] = __float2bfloat16(wi);
  }
}

}  // namespace mptc
