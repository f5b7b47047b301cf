// Completion words and their bounded waits: the memory-order helpers the
// intra dataflow and the scans use.
#pragma once
#include <cstdint>

#include "selection.cuh"

namespace mptc {

// Programmatic dependent launch: the CTAs of a kernel launched that way start while
// the kernel before it in the stream still runs. Every such kernel calls depend() in
// all its threads before it touches global memory: it waits until the kernel before
// has completed with its writes visible, which itself has waited for the one before
// it, so the order is the stream's. A short kernel then lets the next one's CTAs
// start (release_next()) where SMs have room; a long one does not, whose successor's
// waiting CTAs would keep other streams' kernels off the SMs, and releases it as its
// CTAs exit.
__device__ __forceinline__ void depend() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void release_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Completion words are read and written as single 64-bit words, so
// publishing needs no fence and a waiter needs no second load.
__device__ __forceinline__ uint64_t ld_relaxed(const uint64_t *p) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(uint64_t *p, uint64_t v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Waits until done[idx] != 0 and returns the word. Gives up after ~1 s, or at
// once when another wait of this launch already gave up (sets kDevTimeout and
// returns 0), so a broken dependency can never hang the GPU: every later wait
// falls through.
__device__ __forceinline__ uint64_t wait_done(const uint64_t *done, size_t idx, uint32_t *status) {
  uint64_t w = ld_relaxed(done + idx);
  if (w) return w;
  const uint64_t t0 = global_ns();
  for (uint32_t it = 0; it < (1u << 24); ++it) {
    if (it >= 256) __nanosleep(64);  // spin first: the awaited block is usually close
    if ((w = ld_relaxed(done + idx)) != 0) return w;
    if ((it & 63u) == 63u) {
      if (ld_acquire(status) & kDevTimeout) return 0;
      if (global_ns() - t0 > 1000000000ull) break;
    }
  }
  atomicOr(status, kDevTimeout);
  return 0;
}

}  // namespace mptc
