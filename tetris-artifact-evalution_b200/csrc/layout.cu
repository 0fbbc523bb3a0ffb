// Device-side layout transposes between NCHW and NHWC, out of place.
//
// The reference does these on the host through a temporary vector
// (Tetris/tensor_utils.cc:85-111).  Per image both are a 2-D transpose between a [C][H*W] and a
// [H*W][C] matrix.  The kernels are bound by memory: a block moves a tile of 32 channels x 128
// pixels (16 KB) with 16 loads in flight per thread before the first one is used -- a 32 x 32 tile
// with one load per thread and iteration left the memory system half idle (128 x 112 x 112, batch
// 16, there and back: 144 us, 2.8 TB/s).  Pixel rows are moved 128 bytes per warp and access,
// channel rows 16 bytes per lane where the channel count allows it.  The tile's pitch of 129 words
// makes both the row-wise and the column-wise side free of bank conflicts.  Up to 4 and up to 8
// channels (images at the networks' inputs) the tile is 4 x 1024 or 8 x 512, so that its loads are
// as many (3 x 224 x 224, batch 16: 37 us with the 32 x 32 tile, 16.6 with 32 x 128).
#include "internal.h"

namespace tetris {
namespace {

constexpr int kThreads = 256, kElems = 4096;
template <int TC> struct Shape {  // TC channels x TP pixels; pixel rows `pitch` words apart
  static constexpr int TP = kElems / TC, pitch = TP + 32 / TC;
};

// Tile (image, first channel, first pixel) of block `b`: channel tiles fastest, so that blocks that
// run side by side fill whole lines of the channel-innermost side.
struct Tile { size_t img; int c0, p0; };
template <int TC>
__device__ __forceinline__ Tile tile_of(unsigned b, unsigned ctiles, unsigned ptiles, int C, int P) {
  const unsigned r = b / ctiles, n = r / ptiles;
  return {(size_t)n * C * P, (int)(b - r * ctiles) * TC, (int)(r - n * ptiles) * Shape<TC>::TP};
}

// [C][P] -> [P][C] per image.  VEC: 32-channel tiles, C a multiple of 4 and dst 16-byte aligned.
template <int TC, bool VEC>
__global__ void __launch_bounds__(kThreads)
to_channels_last_kernel(const float *src, float *__restrict__ dst, int C, int P, unsigned ctiles, unsigned ptiles) {
  constexpr int TP = Shape<TC>::TP, kPitch = Shape<TC>::pitch;
  __shared__ float tile[TC * kPitch];
  const Tile t = tile_of<TC>(blockIdx.x, ctiles, ptiles, C, P);
  grid_release();
  src = grid_wait(src);
  float v[kElems / kThreads];
#pragma unroll
  for (int i = 0; i < kElems / kThreads; ++i) {
    const int e = threadIdx.x + i * kThreads, c = e / TP, p = e % TP;
    v[i] = t.c0 + c < C && t.p0 + p < P ? __ldcs(src + t.img + (size_t)(t.c0 + c) * P + t.p0 + p) : 0.f;
  }
#pragma unroll
  for (int i = 0; i < kElems / kThreads; ++i) {
    const int e = threadIdx.x + i * kThreads;
    tile[e / TP * kPitch + e % TP] = v[i];
  }
  __syncthreads();
  if (VEC) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = 4 * (lane & 7);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int p = (warp + 8 * i) * 4 + (lane >> 3);
      const float4 w = make_float4(tile[c * kPitch + p], tile[(c + 1) * kPitch + p], tile[(c + 2) * kPitch + p], tile[(c + 3) * kPitch + p]);
      if (t.p0 + p < P && t.c0 + c < C) *reinterpret_cast<float4 *>(dst + t.img + (size_t)(t.p0 + p) * C + t.c0 + c) = w;
    }
  } else {
    // the tile's channels of a pixel are contiguous, and with one channel tile so are its pixels
    const int nc = min(TC, C - t.c0), np = min(TP, P - t.p0);
    const float rcp = 1.f / (float)nc;
    float *o = dst + t.img + (size_t)t.p0 * C + t.c0;
#pragma unroll 4
    for (int i = threadIdx.x; i < nc * np; i += kThreads) {
      const int p = (int)(((float)i + 0.5f) * rcp), c = i - p * nc;  // (exact: i < 4096, nc <= 32)
      o[(size_t)p * C + c] = tile[c * kPitch + p];
    }
  }
}

// [P][C] -> [C][P] per image.  VEC: 32-channel tiles, C a multiple of 4 and src 16-byte aligned.
template <int TC, bool VEC>
__global__ void __launch_bounds__(kThreads)
to_channels_first_kernel(const float *src, float *__restrict__ dst, int C, int P, unsigned ctiles, unsigned ptiles) {
  constexpr int TP = Shape<TC>::TP, kPitch = Shape<TC>::pitch;
  __shared__ float tile[TC * kPitch];
  const Tile t = tile_of<TC>(blockIdx.x, ctiles, ptiles, C, P);
  grid_release();
  src = grid_wait(src);
  if (VEC) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = 4 * (lane & 7);
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int p = (warp + 8 * i) * 4 + (lane >> 3);
      v[i] = t.p0 + p < P && t.c0 + c < C ? __ldcs(reinterpret_cast<const float4 *>(src + t.img + (size_t)(t.p0 + p) * C + t.c0 + c))
                                          : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int p = (warp + 8 * i) * 4 + (lane >> 3);
      tile[c * kPitch + p] = v[i].x; tile[(c + 1) * kPitch + p] = v[i].y;
      tile[(c + 2) * kPitch + p] = v[i].z; tile[(c + 3) * kPitch + p] = v[i].w;
    }
  } else {
    const int nc = min(TC, C - t.c0), np = min(TP, P - t.p0);
    const float rcp = 1.f / (float)nc;
    const float *o = src + t.img + (size_t)t.p0 * C + t.c0;
    float v[kElems / kThreads];
#pragma unroll
    for (int k = 0; k < kElems / kThreads; ++k) {
      const int i = threadIdx.x + k * kThreads, p = (int)(((float)i + 0.5f) * rcp), c = i - p * nc;
      v[k] = i < nc * np ? __ldcs(o + (size_t)p * C + c) : 0.f;
    }
#pragma unroll
    for (int k = 0; k < kElems / kThreads; ++k) {
      const int i = threadIdx.x + k * kThreads, p = (int)(((float)i + 0.5f) * rcp), c = i - p * nc;
      if (i < nc * np) tile[c * kPitch + p] = v[k];
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kElems / kThreads; ++i) {
    const int e = threadIdx.x + i * kThreads, c = e / TP, p = e % TP;
    if (t.c0 + c < C && t.p0 + p < P) dst[t.img + (size_t)(t.c0 + c) * P + t.p0 + p] = tile[c * kPitch + p];
  }
}

template <int TC, bool VEC>
int launch_tiles(const float *src, float *dst, int N, int C, long long P, bool to_last, cudaStream_t st) {
  const long long ctiles = (C + TC - 1) / TC, ptiles = (P + Shape<TC>::TP - 1) / Shape<TC>::TP, blocks = ctiles * ptiles * N;
  if (P >= (1ll << 31) - kElems || blocks >= (1ll << 31)) {
    set_error("layout transpose: shape too large for one launch");
    return TETRIS_ERR_UNSUPPORTED;
  }
  const unsigned b = (unsigned)blocks, ct = (unsigned)ctiles, pt = (unsigned)ptiles;
  TETRIS_CUDA_TRY(launch_overlapped(to_last ? to_channels_last_kernel<TC, VEC> : to_channels_first_kernel<TC, VEC>, dim3(b), kThreads, 0, st, 1,
                                    src, dst, C, (int)P, ct, pt));
  return TETRIS_OK;
}

int launch_transpose(const float *src, float *dst, int N, int C, int H, int W, bool to_last, cudaStream_t st) {
  if (N <= 0) return TETRIS_OK;
  const long long P = (long long)H * W;
  const bool vec = (C & 3) == 0 && (reinterpret_cast<uintptr_t>(to_last ? dst : src) & 15) == 0;
  if (C <= 4) return launch_tiles<4, false>(src, dst, N, C, P, to_last, st);
  if (C <= 8) return launch_tiles<8, false>(src, dst, N, C, P, to_last, st);
  return vec ? launch_tiles<32, true>(src, dst, N, C, P, to_last, st) : launch_tiles<32, false>(src, dst, N, C, P, to_last, st);
}

}  // namespace

int launch_nchw_to_nhwc(const float *src, float *dst, int N, int C, int H, int W, cudaStream_t st) {
  return launch_transpose(src, dst, N, C, H, W, true, st);
}
int launch_nhwc_to_nchw(const float *src, float *dst, int N, int C, int H, int W, cudaStream_t st) {
  return launch_transpose(src, dst, N, C, H, W, false, st);
}

}  // namespace tetris
