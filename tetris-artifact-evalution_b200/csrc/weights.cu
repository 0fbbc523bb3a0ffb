// Weight images of the tensor-core kernels: dense OIHW -> what their loaders copy, for every
// (channel tile, 32-channel chunk, tap), in the swizzled order the tensor core reads.
//
// A block takes the weights of a few output channels and one chunk -- for each channel one
// contiguous run of 32 * KS * KS floats -- through shared memory and writes every image that uses
// them, 16 bytes per thread and store.  (A thread per stored element, gathering its weight from the
// filter and dividing its index apart, took 170 us for the two images of 512 x 512 x 3 x 3.)
#include <cuda_fp16.h>

#include <algorithm>

#include "internal.h"

namespace tetris {
namespace {

constexpr int KC = 32, kThreads = 256;

__device__ __forceinline__ uint32_t round_tf32(float v) { return (__float_as_uint(v) + 0x1000u) & 0xFFFFE000u; }  // (to nearest, ties away)

// Images:
//   tc    split TF32: [chunk][tap][channel tile]{w_hi, w_lo} of bn rows x 32 floats, 16-byte piece j of
//         row r at piece j ^ (r & 7)
//   tc16  split FP16 of w * scale[oc]; plain: [channel tile][chunk][tap] of 128 rows {w_hi[32],
//         w_lo[32]}, piece j of row r at piece j ^ (r & 7); stacked (at most 64 channels): [chunk][tap]
//         of 128 rows of 32, rows 0..63 w_hi and 64..127 w_lo of channel r & 63, piece j at
//         piece j ^ ((r >> 1) & 3)
// Channels past IC or OC are zero.
__global__ void __launch_bounds__(kThreads)
weight_images_kernel(const float *__restrict__ filt, int OC, int IC, int taps, int n_chunks, int R, WeightImages w) {
  extern __shared__ float rows[];  // [R][32 * taps]
  const int chunk = blockIdx.x, oc0 = blockIdx.y * R, run = KC * taps;
  const int have = min(KC, IC - chunk * KC) * taps;
  for (int i = threadIdx.x; i < R * run; i += kThreads) {
    const int r = i / run, e = i - r * run, oc = oc0 + r;
    rows[i] = oc < OC && e < have ? __ldg(filt + ((size_t)oc * IC + chunk * KC) * taps + e) : 0.f;
  }
  __syncthreads();
  if (w.tc16) {
    uint4 *out = static_cast<uint4 *>(w.tc16);
    for (int i = threadIdx.x; i < R * taps * 4; i += kThreads) {  // 8 channels: one piece of w_hi, one of w_lo
      const int piece = i & 3, r = (i >> 2) % R, tap = (i >> 2) / R, oc = oc0 + r;
      const float sc = oc < OC ? w.scale[oc] : 0.f;
      uint32_t hi[4], lo[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float a = rows[r * run + (8 * piece + 2 * e) * taps + tap] * sc, b = rows[r * run + (8 * piece + 2 * e + 1) * taps + tap] * sc;
        const __half2 h = __floats2half2_rn(a, b);
        const float2 f = __half22float2(h);
        const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
        hi[e] = *reinterpret_cast<const uint32_t *>(&h);
        lo[e] = *reinterpret_cast<const uint32_t *>(&l);
      }
      size_t at_hi, at_lo;  // in 16-byte units
      if (w.stack) {
        const size_t image = ((size_t)chunk * taps + tap) * (128 * 4);
        const int j = piece ^ ((oc >> 1) & 3);
        at_hi = image + oc * 4 + j;
        at_lo = image + (oc + 64) * 4 + j;
      } else {
        const size_t row = (((size_t)(oc / 128) * n_chunks + chunk) * taps + tap) * (128 * 8) + (oc % 128) * 8;
        at_hi = row + (piece ^ (oc & 7));
        at_lo = row + ((piece + 4) ^ (oc & 7));
      }
      out[at_hi] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      out[at_lo] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
  }
  if (w.tc) {
    const int tiles = (OC + w.bn - 1) / w.bn;
    for (int i = threadIdx.x; i < R * taps * 8; i += kThreads) {  // 4 channels of w_hi and w_lo
      const int piece = i & 7, r = (i >> 3) % R, tap = (i >> 3) / R, oc = oc0 + r;
      if (oc >= tiles * w.bn) continue;
      uint32_t hi[4], lo[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float v = rows[r * run + (4 * piece + e) * taps + tap];
        hi[e] = round_tf32(v);
        lo[e] = round_tf32(v - __uint_as_float(hi[e]));
      }
      const size_t at = (((size_t)chunk * taps + tap) * tiles + oc / w.bn) * (2 * w.bn * 8) + (oc % w.bn) * 8 + (piece ^ (oc & 7));
      reinterpret_cast<uint4 *>(w.tc)[at] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      reinterpret_cast<uint4 *>(w.tc)[at + w.bn * 8] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
  }
}

}  // namespace

int tensor_prepare(tetris_filter *f, const float *d_dense) {
  WeightImages w;
  int rc;
  if ((rc = conv_tc_prepare(f, d_dense, &w)) || (rc = conv_tc16_prepare(f, d_dense, &w))) return rc;
  if (!w.tc && !w.tc16) return TETRIS_OK;
  const int taps = f->kernel_size * f->kernel_size, n_chunks = (f->in_channel + KC - 1) / KC;
  int R = 16;  // rows of a block: at most 48 KB of shared memory
  while (R * KC * taps * 4 > 48 * 1024) R /= 2;
  const int rows = f->out_channel <= 64 ? 64 : (f->out_channel + 127) / 128 * 128;  // padded to whole channel tiles
  weight_images_kernel<<<dim3((unsigned)n_chunks, (unsigned)(rows / R)), kThreads, (size_t)R * KC * taps * 4>>>(
      d_dense, f->out_channel, f->in_channel, taps, n_chunks, R, w);
  TETRIS_CUDA_TRY(cudaGetLastError());
  return TETRIS_OK;
}

}  // namespace tetris
