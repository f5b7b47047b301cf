// The kernels' refit from integer sums (refit_quick, candidate_eval.cuh, compiled here
// for the host) against their float steps (refit_exact): wherever the first claims to
// be sure, all six snapped endpoints are the second's, and the two computations stay
// within the margin that the claim rests on. Arguments: seed, blocks.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

// ---- what the header uses of CUDA -------------------------------------------------
#define __device__
#define __forceinline__ inline
#define __align__(n) __attribute__((aligned(n)))
using std::max;
struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
struct uint2 { uint32_t x, y; };
struct alignas(16) uint4 { uint32_t x, y, z, w; };
struct Dim { unsigned x; };
static const Dim threadIdx{0}, blockDim{1};
inline float2 make_float2(float x, float y) { return {x, y}; }
inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }
inline uint2 make_uint2(uint32_t x, uint32_t y) { return {x, y}; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fdiv_rn(float a, float b) { return a / b; }
inline float __frcp_rn(float a) { return 1.0f / a; }
inline float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
inline float __fadd_rd(float a, float b) {
  const double d = (double)a + (double)b;
  const float f = (float)d;
  return (double)f > d ? std::nextafterf(f, -INFINITY) : f;
}
inline int __float2int_rz(float a) {
  return a != a ? 0 : a >= 2147483648.0f ? INT32_MAX : a < -2147483648.0f ? INT32_MIN : (int)a;
}
inline float __uint2float_rn(uint32_t a) { return (float)a; }
inline uint32_t __float_as_uint(float a) {
  uint32_t u;
  std::memcpy(&u, &a, 4);
  return u;
}
inline uint32_t __byte_perm(uint32_t a, uint32_t b, uint32_t s) {
  const uint64_t v = (uint64_t)b << 32 | a;
  uint32_t r = 0;
  for (int i = 0; i < 4; ++i) r |= (uint32_t)(v >> (8 * (s >> (4 * i) & 7u)) & 0xFFu) << (8 * i);
  return r;
}
inline uint32_t __dp4a(uint32_t a, uint32_t b, uint32_t c) {
  for (int i = 0; i < 4; ++i) c += (a >> (8 * i) & 0xFFu) * (b >> (8 * i) & 0xFFu);
  return c;
}
template <class T> T __ldg(const T *p) { return *p; }
// of the parts that need a warp, which are not called here
inline uint32_t __shfl_sync(uint32_t, uint32_t v, int) { return v; }
inline int __reduce_add_sync(uint32_t, int v) { return v; }
inline void __syncwarp() {}

#include "candidate_eval.cuh"

using namespace mptc;

static uint64_t g_state;
static uint32_t rnd() {  // xorshift64*
  g_state ^= g_state >> 12;
  g_state ^= g_state << 25;
  g_state ^= g_state >> 27;
  return (uint32_t)(g_state * 2685821657736338717ull >> 32);
}

static void random_block(PixBlocks<1> &px) {
  const uint32_t mode = rnd() % 7;  // noise, narrow to wide ranges, near white, few levels, one odd pixel
  const int span[7] = {256, 3, 9, 40, 100, 2, 1};
  uint8_t v[3][16];
  for (auto &ch : v) {
    const int base = mode == 0 ? 0 : (int)(rnd() % 256);
    for (auto &p : ch) p = (uint8_t)std::min(255, std::max(0, base + (int)(rnd() % span[mode]) - span[mode] / 2));
    if (mode == 5)
      for (auto &p : ch) p = (uint8_t)(rnd() % 3 ? 255 - rnd() % 3 : 21 * (rnd() % 13));
    if (mode == 6) ch[rnd() % 16] = (uint8_t)rnd();
  }
  std::memset(&px, 0, sizeof px);
  for (int c = 0; c < 3; ++c)
    for (int i = 0; i < 16; ++i) {
      px.w[c][0][i / 4] |= (uint32_t)v[c][i] << (8 * (i % 4));
      px.w[3][0][c] += v[c][i];
      px.w[3][0][3] += v[c][i] * v[c][i];
    }
}

static uint32_t random_word() {
  uint32_t w = rnd();
  const uint32_t kind = rnd() % 6, base = (rnd() & 3u) * 0x55555555u;
  if (kind == 1 || kind == 2) {  // all but one to three indices equal: the largest finite f
    w = base;
    for (uint32_t n = kind == 1 ? 1 : 1 + rnd() % 3; n; --n) {
      const uint32_t p = 2 * (rnd() % 16);
      w = (w & ~(3u << p)) | (rnd() & 3u) << p;
    }
  } else if (kind == 3) {
    w &= 0xAAAAAAAAu;
  } else if (kind == 4) {
    w |= 0xAAAAAAAAu;
  }
  return w;
}

int main(int argc, char **argv) {
  g_state = 88172645463325252ull + 7919ull * (argc > 1 ? std::strtoull(argv[1], nullptr, 10) : 1);
  const long blocks = argc > 2 ? std::atol(argv[2]) : 100000;
  float4 wk[4];
  for (uint32_t k = 0; k < 4; ++k) {
    const float order = k == 0 ? 0.f : k == 1 ? 3.f : k == 2 ? 1.f : 2.f, a = (3.0f - order) / 3.0f, b = order / 3.0f;
    wk[k] = make_float4(a * a, b * b, a * b, 0.f);
  }
  static SnapTables st;
  build_snap_edges(st);
  const float third = 1.0f / 3.0f;
  long pairs = 0, sure = 0, degenerate = 0, wrong = 0;
  double worst = 0;
  for (long n = 0; n < blocks; ++n) {
    PixBlocks<1> px;
    random_block(px);
    const PixBlock<1> t{px, 0};
    for (int rep = 0; rep < 16; ++rep, ++pairs) {
      const uint32_t word = random_word();
      const WeightSums ws = weight_sums(word, wk);
      RefitValues q, x;
      const bool ok = refit_quick(t, st, word, ws, q);
      refit_exact(t, st, word, ws, x);
      uint32_t eq, ex;
      const int dq = refit_error(t, q, word, 100, eq), dx = refit_error(t, x, word, 100, ex);
      bool same = dq == dx && eq == ex;
      for (int i = 0; i < 6; ++i) same = same && (q.snap[i] & 0xFFu) == (x.snap[i] & 0xFFu);
      sure += ok;
      if (ok && !same && ++wrong <= 5) std::printf("word %08x: %d %d, endpoints %08x %08x\n", word, dq, dx, eq, ex);
      // the endpoints before snapping, both ways, and the margin
      const uint32_t tmax = max(px.w[3][0][0], max(px.w[3][0][1], px.w[3][0][2]));
      const double margin = (double)kRefitRel * tmax * std::fabs(ws.f) * std::max(ws.asq, ws.bsq) + kRefitAbs;
      if (!(margin < 0.25)) {
        ++degenerate;
        if (ok) ++wrong;
        continue;
      }
      for (int c = 0; c < 3; ++c) {
        float ax = 0, bx = 0;
        uint32_t S = 0;
        for (int i = 0; i < 16; ++i) {
          const uint32_t k = word >> (2 * i) & 3u, p = px.w[c][0][i / 4] >> (8 * (i % 4)) & 0xFFu;
          const uint32_t order = k == 0 ? 0 : k == 1 ? 3 : k == 2 ? 1 : 2;
          ax += (float)p * ((3.0f - (float)order) / 3.0f);
          bx += (float)p * ((float)order / 3.0f);
          S += p * order;
        }
        const float b = (float)S * third, a = (float)(3 * px.w[3][0][c] - S) * third;
        const float p1 = ws.f * (ax * ws.bsq - bx * ws.ab) + 0.5f, p2 = ws.f * (bx * ws.asq - ax * ws.ab) + 0.5f;
        const float v1 = std::fmaf(ws.f, a * ws.bsq - b * ws.ab, 0.5f), v2 = std::fmaf(ws.f, b * ws.asq - a * ws.ab, 0.5f);
        if (std::fabs(p1) < 260) worst = std::max(worst, std::fabs((double)p1 - v1) / margin);
        if (std::fabs(p2) < 260) worst = std::max(worst, std::fabs((double)p2 - v2) / margin);
      }
    }
  }
  std::printf("pairs %ld unsure %.3f%% degenerate %.3f%% wrong %ld largest difference %.3f of the margin\n", pairs,
              100.0 * (pairs - sure) / pairs, 100.0 * degenerate / pairs, wrong, worst);
  return wrong == 0 && worst < 1.0 && sure > pairs / 2 ? 0 : 1;
}
