// Launches with programmatic stream serialization, for kernels that call depend()
// (completion.cuh) before they touch global memory.
#pragma once
#include <cuda_runtime.h>

namespace mptc {

// Behind the kernel before it in the stream. Used inside a frame's chain of kernels,
// not behind an event wait. A frame is a chain of some 13 kernels of 3 to 20 us;
// launched this way, with the work area zeroed by the first of them instead of two
// memsets, an inter frame takes 212 us at 1080p (245 before) and 74.5 us at 256x256
// (107).
template <typename... Par, typename... Arg>
void launch_if_chained(bool chained, void (*kernel)(Par...), dim3 grid, int threads, size_t smem, cudaStream_t s,
                       Arg... arg) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = chained ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, Par(arg)...);
}
template <typename... Par, typename... Arg>
void launch_chain_smem(void (*kernel)(Par...), dim3 grid, int threads, size_t smem, cudaStream_t s, Arg... arg) {
  launch_if_chained(true, kernel, grid, threads, smem, s, arg...);
}

template <typename... Par, typename... Arg>
void launch_chain(void (*kernel)(Par...), dim3 grid, int threads, cudaStream_t s, Arg... arg) {
  launch_chain_smem(kernel, grid, threads, 0, s, arg...);
}

// The first kernel of a call, behind whatever the caller has queued: the same
// outside a capture, a plain launch within one, where the stream's edge may join
// several streams.
template <typename... Par, typename... Arg>
void launch_after(void (*kernel)(Par...), dim3 grid, int threads, cudaStream_t s, Arg... arg) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) != cudaSuccess) {
    cudaGetLastError();  // the launch itself reports what is wrong
    st = cudaStreamCaptureStatusActive;
  }
  launch_if_chained(st == cudaStreamCaptureStatusNone, kernel, grid, threads, 0, s, arg...);
}

}  // namespace mptc
