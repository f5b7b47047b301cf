// C ABI of the endpoint transform and of the GPU decoder (include/mptc_gb300.h).
#include <cuda_runtime.h>

#include <new>
#include <string>

#include "../../include/mptc_gb300.h"
#include "endpoint_codec.cuh"
#include "launch.cuh"

namespace {

bool tiled_size(int32_t width, int32_t height) {
  return width > 0 && height > 0 && width % 256 == 0 && height % 256 == 0 &&
         (int64_t)(width / 4) * (height / 4) <= (int64_t)1 << 30;
}

}  // namespace

struct mptc_decoder {
  int width = 0, height = 0, bw = 0, bh = 0, nblk = 0, sa = 0, ntiles = 0;
  uint64_t *link = nullptr;   // [nblk] index words and copies
  uint64_t *state = nullptr;  // [ntiles] of the unique blocks' scan, zero between frames; then its tile counter
  uint8_t *planes = nullptr;  // [6][nblk] decoded endpoint planes
  uint32_t *flags = nullptr;  // device error flags, status bits
  bool state_lost = false;    // a frame's second kernel, which zeroes the state, was not launched
  std::string err;
};

namespace {

mptc_status dfail(mptc_decoder *d, mptc_status st, const std::string &msg) {
  if (d) d->err = msg;
  return st;
}

void release(mptc_decoder *d) {
  cudaFree(d->link);
  cudaFree(d->state);
  cudaFree(d->planes);
  cudaFree(d->flags);
}

}  // namespace

extern "C" {

mptc_status mptc_endpoint_coefficients(int32_t width, int32_t height, const uint64_t *blocks_dev,
                                       uint8_t *coeff_dev, void *stream) {
  if (!tiled_size(width, height) || !blocks_dev || !coeff_dev) return MPTC_EINVAL;
  const int bw = width / 4, bh = height / 4;
  const dim3 grid(bw / mptc::kTile, bh / mptc::kTile, 6);
  mptc::launch_after(mptc::endpoint_forward_kernel, grid, mptc::kCodecThreads, (cudaStream_t)stream, blocks_dev, bw, bh,
                     coeff_dev);
  return cudaGetLastError() == cudaSuccess ? MPTC_OK : MPTC_ECUDA;
}

mptc_status mptc_decoder_create(int32_t width, int32_t height, int32_t search_area, mptc_decoder **out) {
  if (!out || !tiled_size(width, height) || search_area < 1 || search_area > 63) return MPTC_EINVAL;
  mptc_decoder *d = new (std::nothrow) mptc_decoder();
  if (!d) return MPTC_ENOMEM;
  d->width = width;
  d->height = height;
  d->bw = width / 4;
  d->bh = height / 4;
  d->nblk = d->bw * d->bh;
  d->sa = search_area;
  d->ntiles = (d->nblk + mptc::kScanTile - 1) / mptc::kScanTile;
  const size_t n = (size_t)d->nblk;
  const size_t state_bytes = ((size_t)d->ntiles + 1) * sizeof(uint64_t);
  cudaError_t e = cudaMalloc(&d->link, n * sizeof(uint64_t));
  if (e == cudaSuccess) e = cudaMalloc(&d->state, state_bytes);
  if (e == cudaSuccess) e = cudaMemset(d->state, 0, state_bytes);
  if (e == cudaSuccess) e = cudaMalloc(&d->planes, 6 * n);
  if (e == cudaSuccess) e = cudaMalloc(&d->flags, 2 * sizeof(uint32_t));
  if (e == cudaSuccess) e = cudaMemset(d->flags, 0, 2 * sizeof(uint32_t));
  // every link a word from the start: whatever a block reads leads to a word
  if (e == cudaSuccess) e = cudaMemset(d->link, 1, n * sizeof(uint64_t));
  // the memsets are queued, and no other stream's first frame waits for them
  if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);
  if (e != cudaSuccess) {
    release(d);
    delete d;
    return e == cudaErrorMemoryAllocation ? MPTC_ENOMEM : MPTC_ECUDA;
  }
  *out = d;
  return MPTC_OK;
}

mptc_status mptc_decoder_destroy(mptc_decoder *d) {
  if (!d) return MPTC_EINVAL;
  release(d);
  delete d;
  return MPTC_OK;
}

mptc_status mptc_decode_frame(mptc_decoder *d, const uint8_t *coeff_dev, const uint8_t *motion_dev,
                              const uint32_t *unique_dev, uint32_t n_unique, const uint64_t *prev_dev,
                              uint64_t *out_dev, void *stream) {
  if (!d) return MPTC_EINVAL;
  if (!coeff_dev || !motion_dev || !out_dev || (n_unique && !unique_dev))
    return dfail(d, MPTC_EINVAL, "decode_frame: NULL buffer");
  if (n_unique > (uint32_t)d->nblk) return dfail(d, MPTC_EINVAL, "decode_frame: more unique entries than blocks");
  cudaStream_t s = (cudaStream_t)stream;
  const int tiles = (d->bw / mptc::kTile) * (d->bh / mptc::kTile);
  uint32_t *claim = reinterpret_cast<uint32_t *>(d->state + d->ntiles);
  if (d->state_lost) {
    const cudaError_t z = cudaMemsetAsync(d->state, 0, ((size_t)d->ntiles + 1) * sizeof(uint64_t), s);
    if (z != cudaSuccess) return dfail(d, MPTC_ECUDA, cudaGetErrorString(z));
    d->state_lost = false;
  }
  mptc::launch_after(mptc::decode_parts_kernel, d->ntiles + 6 * tiles, mptc::kCodecThreads, s, coeff_dev, d->bw, d->bh,
                     d->planes, motion_dev, prev_dev, d->sa, unique_dev, n_unique, d->ntiles, d->state, claim, d->link,
                     d->flags, d->flags + 1);
  mptc::launch_chain(mptc::decode_link_kernel, (d->nblk + 255) / 256, 256, s, d->planes, d->nblk, d->link, d->state,
                     d->ntiles, claim, out_dev);
  const cudaError_t e = cudaGetLastError();
  d->state_lost = e != cudaSuccess;
  return e == cudaSuccess ? MPTC_OK : dfail(d, MPTC_ECUDA, cudaGetErrorString(e));
}

mptc_status mptc_decoder_check(mptc_decoder *d, void *stream, uint32_t *flags) {
  if (!d) return MPTC_EINVAL;
  uint32_t w[2] = {0, 0};
  cudaError_t e = cudaMemcpyAsync(w, d->flags, sizeof(w), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(d->flags, 0, sizeof(w), (cudaStream_t)stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
  if (e != cudaSuccess) return dfail(d, MPTC_ECUDA, cudaGetErrorString(e));
  const uint32_t h = w[0];
  if (flags) *flags = h;
  if (w[1] & mptc::kDevTimeout) return dfail(d, MPTC_ETIMEOUT, "device-side dependency wait expired");
  if (w[1] & mptc::kDevBadScan) return dfail(d, MPTC_ESTATE, "a frame began before the one before it had ended");
  if (h) {
    std::string m = "decoded frames held";
    if (h & mptc::kDecBadRef) m += " motion codes that copy from outside the frame or from undecoded blocks";
    if (h & mptc::kDecBadUnique) m += (h & mptc::kDecBadRef) ? " and" : "", m += " a unique count that differs from the palette";
    return dfail(d, MPTC_EINVAL, m);
  }
  return MPTC_OK;
}

const char *mptc_decoder_last_error(const mptc_decoder *d) { return d ? d->err.c_str() : "null decoder"; }

}  // extern "C"
