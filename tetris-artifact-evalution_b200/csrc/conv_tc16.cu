// Dense contraction on the 5th-generation tensor cores in SPLIT FP16: the fast variant of the
// layers with 8 or more input channels (tcgen05.mma kind::f16 + TMEM + TMA).
//
// Arithmetic.  x' = 16 x = x_hi + x_lo and w' = w * 2^sh = w_hi + w_lo with *_hi the value rounded
// to FP16 (11 significant bits) and *_lo the FP16-rounded remainder; D += w_hi*x_hi + w_hi*x_lo +
// w_lo*x_hi in FP32 accumulators, scaled back by 2^-sh / 16 (exact) at the store; sh is chosen per
// OUTPUT CHANNEL, so channels of very different magnitude keep their own full precision.  The
// products are exact in FP32; what is dropped is w_lo*x_lo and the rounding of the remainders,
// about 2^-22 of a product each -- the same as the split-TF32 variant (conv_tc.cu), at twice the
// tensor-core rate.  sh puts a channel's largest |w'| at about 2^13.
//
// Range.  FP16 has a window: |x| < 2048 after the fixed scale, absolute error of at most 2e-9 per
// activation.  The converter warps of a CTA record the largest |x| they see; a CTA that finds it
// outside [2^-8, 2048) runs its work items again with a scale taken from that maximum and the
// activations cut into two bands, the upper one of 16 binades, with a pass over K per band, whose sums
// are added up in FP32; where activations lie below 32 binades, a last time with three bands.  No second launch and no state between launches: what a CTA
// recomputes is its own output.
//
// The tensor core truncates when it adds into its FP32 accumulator, so the accumulation chain is
// cut every 1 to 8 K steps of 6 MMAs (4 on stacked tiles; see partial_steps): the tensor core accumulates
// from zero into one of two partial accumulators and CUDA-core warps add the partials to a running sum
// in registers.
//
// Structure.  D[channel][pixel]: the M side is 128 output channels (the weights), the N side up to
// 256 output pixels (the activations), K = (32-channel chunk, filter tap).  Both operands are read
// from shared memory.  Why this way round and this size: an MMA of M = 128 reads 128 x 32 bytes of
// A and N x 32 bytes of B from shared memory (128 bytes/clock) and computes for N/2 clocks, so
// N = 128 needs the whole shared-memory pipe while N = 256 leaves a quarter of it for the weight
// copies and the conversion; with the weights on the M side one 16 KB weight image serves 256
// pixels (L2 -> SM weight traffic halved against 128-pixel tiles), and an accumulator row is an
// output channel, so a warp turns 16 pixels x 32 consecutive channels over in a small staging block, from
// where TMA stores carry 8 pixels at a time on, or, where the channel count is no multiple of 4 or the
// output not 16-byte aligned, the warp itself, a pixel's 32 channels as one line.
//   * warp 0 (one thread): TMA loads of activation patches (tile + halo, 32 channels, out-of-range
//     coordinates zero-filled = the padding) and bulk copies of weight images, each into a ring;
//   * converter warps: a landed patch, once, in place: each 128-byte row of 32 FP32 channels
//     becomes {x_hi[32], x_lo[32]} FP16;
//   * warp 1 (one elected lane): the MMAs.  The B operand of a tap is a WINDOW of the converted
//     patch: a descriptor whose start is shifted by the tap's (row, column) and whose 8-pixel
//     groups are one patch row apart.  The 128-byte swizzle is a function of the shared-memory
//     address, so a window that starts at any 128-byte row reads back what TMA wrote;
//   * eight summing warps: partial accumulators -> running sums -> global memory.
// At stride S the input splits into S x S phases; each phase is a patch of its own (TMA element
// strides) whose taps read it at stride 1, so a phase is loaded and converted once per chunk.
// Filters with at most 64 output channels stack {w_hi, w_lo} on the M side: one MMA multiplies
// both halves, 4 MMAs per K step instead of 6; the halves are added in the epilogue.
// Few tiles (small batches, deep layers): the K range of a tile is cut over a cluster of up to 8
// CTAs, whose sums meet in distributed shared memory and are added in slice order (bit-reproducible,
// no zeroing of the output, ReLU-fusable).
// Every barrier wait is bounded; on a timeout an error flag is raised, all roles drain, TMEM is
// freed and the kernel returns; the host reports TETRIS_ERR_CUDA.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <new>

#include "internal.h"

namespace tetris {
namespace {

constexpr int BM = 128, KC = 32;         // channels of a tile; K chunk (32 input channels)
constexpr int kTW = 8;                   // a pixel group is 8 consecutive output columns
constexpr int kXStagesMax = 6, kWStagesMax = 8;
constexpr int kSumWarps = 8;
constexpr int kBandBits = 16;            // banded passes: bands of 16 binades below the largest activation
// Per summing warp: two blocks of 16 pixels x 32 channels on their way to the output, and for
// stacked tiles 32 pixels x 32 accumulator lanes handed to the warp with the other half.
__host__ __device__ constexpr int stage_bytes(bool stack) { return kSumWarps * (4096 + (stack ? 4096 : 0)); }
constexpr int kNumBars = 3 * kXStagesMax + 2 * kWStagesMax + 6;  // (even: what follows is read 16 bytes at a time)
constexpr uint32_t kSpinLimit = 1u << 22;
constexpr float kXScale = 16.f;          // activations are multiplied by this before the split (undone in out_scale)

enum { kLinear = 0, kFlat = 1, kGrid = 2 };

// Division of 0 <= n < 2^31 by a launch constant: q = (umulhi(n, mul) + n) >> shift with
// shift = ceil(log2 d) and mul = floor(2^32 (2^shift - d) / d) + 1 (the items' coordinates are worked
// out by every role; an integer division costs a warp ~100 clocks).
struct FastDiv {
  uint32_t d, mul, shift;
};
FastDiv fast_div(uint32_t d) {
  FastDiv f;
  f.d = d; f.shift = 0;
  while ((1ull << f.shift) < d) ++f.shift;
  f.mul = (uint32_t)(((1ull << 32) * ((1ull << f.shift) - d)) / d + 1);
  return f;
}
__device__ __forceinline__ int quot(int n, const FastDiv &f) { return (int)((__umulhi((uint32_t)n, f.mul) + (uint32_t)n) >> f.shift); }

struct Tc16Params {
  float *out;
  int N, OH, OW, OC, S, P, KS;
  int mode;                    // kLinear: 1x1 filters at stride 1, a tile is `npx` consecutive pixels of the batch;
                               // kFlat: `npx` consecutive positions of one image laid out with its padded width PW
                               // (positions past OW in a row are computed and dropped);
                               // kGrid: 8 columns x TH rows x NB images
  int npx;                     // pixels of a tile = N of the MMAs, a multiple of 16
  int PW;                      // patch width in pixels
  int PHI;                     // patch rows of one image
  int TH, NB;                  // kGrid: output rows and images of a tile
  int box_rows;                // 128-byte rows a patch load delivers
  int x_stage_bytes, n_x, n_w;
  int tiles_w, tiles_h, tiles_n, oc_tiles, total_tiles;
  FastDiv by_oc_tiles, by_tiles_w, by_tiles_h, by_PW, by_PHI;
  int super;                   // K steps per partial sum (a power of two)
  int n_chunks;
  int d;                       // CTAs of a cluster = slices of a tile's K range
  int relu;                    // max(y, 0) at the store
  int tma_store;               // pixel groups leave through TMA stores (channel count and alignment allow it)
  long long total_pixels;      // N * OH * OW
  const float *out_scale;      // per output channel: 2^-sh[oc] / 16 (undoes the weight and activation scaling)
  int *error_flag;
  const __half *w_tiles;
  unsigned spin_limit;         // polls after which a barrier wait gives up (0: kSpinLimit)
  int withhold_first_load;     // failure-detection test only: every CTA leaves out its first activation load
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// (does not suspend the thread: for the loader, which polls two rings)
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded wait.  Gives up when the limit (abort_flag[1]) is hit or when another role already gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint32_t limit = (uint32_t)abort_flag[1];
  for (uint32_t i = 1; i < limit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 63) == 63) {
      if (*abort_flag) return false;
      __nanosleep(32);
    }
  }
  *abort_flag = 1;
  return false;
}
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}
// After a give-up: wait (bounded, whatever the abort flag says) for an asynchronous operation this
// thread started earlier, so that the CTA does not leave while a copy into its shared memory or
// an MMA on its tensor memory is still in flight.
__device__ __forceinline__ void mbar_drain(uint32_t bar, uint32_t parity) {
  for (uint32_t i = 0; i < (1u << 16); ++i) {
    if (mbar_try_wait(bar, parity)) return;
    if ((i & 63) == 63) __nanosleep(64);
  }
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// K-major operand; 8-row groups `sbo_bytes` apart; layout 2 = 128-byte rows with the 128B swizzle,
// 4 = 64-byte rows with the 64B swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t sbo_bytes, uint32_t layout) {
  return (uint64_t)((saddr >> 4) & 0x3FFF) | (1ull << 16) | ((uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32) | (1ull << 46) |
         ((uint64_t)layout << 61);
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(pred));
  return pred != 0;
}
// D[tmem] (+)= A[smem] * B[smem], FP16 operands, FP32 accumulate.  The descriptors are passed as
// words: the high ones are constants, the low ones a start address plus a constant.
__device__ __forceinline__ void umma_f16_ss(uint32_t tmem_d, uint32_t da_lo, uint32_t da_hi, uint32_t db_lo, uint32_t db_hi,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n.reg .pred p;\n.reg .b64 da, db;\nmov.b64 da, {%1, %2};\nmov.b64 db, {%3, %4};\nsetp.ne.b32 p, %6, 0;\n"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n}"
               ::"r"(tmem_d), "r"(da_lo), "r"(da_hi), "r"(db_lo), "r"(db_hi), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                 "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
                 "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ float pow2f(int e) { return __uint_as_float((uint32_t)(min(127, max(-126, e)) + 127) << 23); }
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {  // `addr` of this CTA in CTA `rank` of the cluster
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
// Pixels of a tile that one CTA of a cluster of `d` adds up and stores: whole blocks of 16.
__host__ __device__ constexpr int share_pixels(int npx, int d) { return ((npx >> 4) + d - 1) / d * 16; }

// One 128-byte row of a patch, in place: 32 FP32 channels, each through `scaled`, to {x_hi[32], x_lo[32]} FP16.
// `look` sees the 16-byte pieces before.
template <typename F, typename G>
__device__ __forceinline__ void convert_row(float4 *rp, int swz, F scaled, G look) {
  float4 v[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) v[c] = rp[c ^ swz];
  uint32_t hi[16], lo[16];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    look(v[c]);
    const float x[4] = {scaled(v[c].x), scaled(v[c].y), scaled(v[c].z), scaled(v[c].w)};
    const __half2 h01 = __floats2half2_rn(x[0], x[1]), h23 = __floats2half2_rn(x[2], x[3]);
    const float2 f01 = __half22float2(h01), f23 = __half22float2(h23);
    hi[2 * c] = *reinterpret_cast<const uint32_t *>(&h01);
    hi[2 * c + 1] = *reinterpret_cast<const uint32_t *>(&h23);
    lo[2 * c] = pack_half2(x[0] - f01.x, x[1] - f01.y);
    lo[2 * c + 1] = pack_half2(x[2] - f23.x, x[3] - f23.y);
  }
  uint4 *wp = reinterpret_cast<uint4 *>(rp);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    wp[c ^ swz] = make_uint4(hi[4 * c], hi[4 * c + 1], hi[4 * c + 2], hi[4 * c + 3]);
    wp[(c + 4) ^ swz] = make_uint4(lo[4 * c], lo[4 * c + 1], lo[4 * c + 2], lo[4 * c + 3]);
  }
}

// The same in the passes behind the first, which few launches make: out of line, so that the first one's code and
// registers stay as they are (inlined, the smallest launches took 2 % longer: 64->64 3x3 at 56x56, one image).
// band < 0: all of it, `seen` becomes the bits of the largest finite |activation|.  band 0: what is not below `lo`
// (infinities and NaN with it).  band > 0: what lies in [lo, hi); `seen` becomes 2 * bits - 1 of the smallest
// |activation|, zeros last.
__device__ __noinline__ unsigned convert_row_again(uint32_t saddr, int swz, float scale, float lo, float hi, unsigned seen, int band) {
  float4 *rp = static_cast<float4 *>(__cvta_shared_to_generic(saddr));
  auto nothing = [](const float4 &) {};
  if (band < 0)
    convert_row(rp, swz, [&](float x) {
      if (fabsf(x) < __int_as_float(0x7F800000)) seen = max(seen, __float_as_uint(fabsf(x)));
      return x * scale;
    }, nothing);
  else if (band == 0)
    convert_row(rp, swz, [&](float x) { return fabsf(x) < lo ? 0.f : x * scale; }, nothing);
  else
    convert_row(rp, swz, [&](float x) {
      seen = min(seen, 2u * __float_as_uint(x) - 1u);
      return fabsf(x) < hi && !(fabsf(x) < lo) ? x * scale : 0.f;
    }, nothing);
  return seen;
}

// Sums of a lane in tensor memory, multiplied by f.
__device__ __noinline__ void scale_columns(uint32_t taddr, int ncols, float f) {
#pragma unroll 1
  for (int c0 = 0; c0 < ncols; c0 += 16) {
    uint32_t v[16];
    tmem_ld16(taddr + c0, v);
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * f);
    tmem_st16(taddr + c0, v);
  }
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// NMAX: most pixels of a tile.  A summing warp keeps NMAX / 2 running sums per thread, which sets
// the register count: 12 warps (2 of them converters) for 256 pixels, 16 warps (6 converters) for
// 128.  STACK: at most 64 output channels, {w_hi, w_lo} stacked on the M side.
// The 256-pixel instances spill: 168 registers a thread hold 128 running sums, and ptxas reports 32 (stacked 64)
// bytes of spill stores and 52 (100) of loads.
template <int NMAX> struct Roles {
  static constexpr int kConv = NMAX == 256 ? 2 : 6;
  static constexpr int kFirstSum = 2 + kConv;
  static constexpr int kThreads = 32 * (kFirstSum + kSumWarps);
};

template <int NMAX, bool STACK>
__global__ void __launch_bounds__(Roles<NMAX>::kThreads, 1)
conv_tc16_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_out, const Tc16Params p) {
  constexpr int kConv = Roles<NMAX>::kConv, kFirstSum = Roles<NMAX>::kFirstSum, kThreads = Roles<NMAX>::kThreads;
  constexpr int kWBytes = STACK ? 8192 : 16384;   // weights of one K step
  constexpr int kOcTile = STACK ? 64 : 128;       // output channels of a tile
  constexpr int NC = NMAX / 2;                    // running sums (pixels) per summing thread, at most
  constexpr int kTmemCols = 2 * NMAX;             // two partial accumulators
  extern __shared__ unsigned char smem_raw[];
  unsigned char *xbase = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  unsigned char *wbase = xbase + (size_t)p.n_x * p.x_stage_bytes;
  unsigned char *exch = wbase + (size_t)p.n_w * kWBytes;
  uint64_t *bars = reinterpret_cast<uint64_t *>(exch + stage_bytes(STACK));
  int4 *gtabs = reinterpret_cast<int4 *>(bars + kNumBars);  // per summing warp: where each of its 8-pixel groups goes
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(gtabs + kSumWarps * (NC / 8));
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  unsigned *seen_slot = tmem_slot + 3;            // largest |activation| of this CTA, FP32 bits
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto bar_xfull = [&](int s) { return smem_u32(&bars[s]); };
  auto bar_xconv = [&](int s) { return smem_u32(&bars[kXStagesMax + s]); };
  auto bar_xempty = [&](int s) { return smem_u32(&bars[2 * kXStagesMax + s]); };
  auto bar_wfull = [&](int s) { return smem_u32(&bars[3 * kXStagesMax + s]); };
  auto bar_wempty = [&](int s) { return smem_u32(&bars[3 * kXStagesMax + kWStagesMax + s]); };
  auto bar_pfull = [&](int b) { return smem_u32(&bars[kNumBars - 6 + b]); };
  auto bar_pempty = [&](int b) { return smem_u32(&bars[kNumBars - 4 + b]); };
  auto bar_drain = [&]() { return smem_u32(&bars[kNumBars - 2]); };

  if (tid == 0) {
    for (int s = 0; s < kXStagesMax; ++s) { mbar_init(bar_xfull(s), 1); mbar_init(bar_xconv(s), kConv); mbar_init(bar_xempty(s), 1); }
    for (int s = 0; s < kWStagesMax; ++s) { mbar_init(bar_wfull(s), 1); mbar_init(bar_wempty(s), 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(bar_pfull(b), 1); mbar_init(bar_pempty(b), kSumWarps); }
    mbar_init(bar_drain(), 1);
    abort_flag[0] = 0;
    abort_flag[1] = (int)(p.spin_limit ? p.spin_limit : kSpinLimit);
    *seen_slot = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  if (tid == 0) grid_release();  // (this CTA has its tensor memory: nothing it waits for can be held by the next launch)
  if (warp != 0) grid_wait();    // (warp 0 sends for weights first)

  // Work items: tile blockIdx.x / d, + gridDim.x / d, ... (d > 1: exactly one).  The channel tile
  // is the fastest index, so CTAs that run side by side read the same activation patch.
  const int rank = p.d > 1 ? (int)(blockIdx.x % p.d) : 0;
  const int tile0 = blockIdx.x / p.d, tile_step = gridDim.x / p.d;
  const int chunk0 = p.n_chunks * rank / p.d, chunk1 = p.n_chunks * (rank + 1) / p.d;
  const int taps = p.KS * p.KS;
  const int iters = taps * (chunk1 - chunk0);       // K steps of an item (per band)
  const int supers = (iters + p.super - 1) / p.super;
  const int phases = min(p.S, p.KS);                // input phases per axis that a tap falls into
  auto decode = [&](int t, int &oc0, int &w0, int &h0, int &n0) {
    int u = quot(t, p.by_oc_tiles);
    oc0 = (t - u * p.oc_tiles) * kOcTile;
    t = quot(u, p.by_tiles_w);
    w0 = u - t * p.tiles_w;                         // kLinear, kFlat: number of the tile; kGrid: tile column
    u = quot(t, p.by_tiles_h);
    h0 = (t - u * p.tiles_h) * p.TH;
    n0 = u * p.NB;
  };
  // output pixel of column j of a tile, -1 where it is none
  auto pixel_of = [&](int j, int w0, int h0, int n0) -> int {
    if (p.mode == kLinear) {
      const long long px = (long long)w0 * p.npx + j;
      return px < p.total_pixels ? (int)px : -1;
    }
    int oh, ow, n = n0;
    bool in = true;
    if (p.mode == kFlat) {
      const int pos = w0 * p.npx + j;
      oh = quot(pos, p.by_PW); ow = pos - oh * p.PW;
    } else {
      const int g = j >> 3, i = p.NB > 1 ? quot(g, p.by_PHI) : 0;
      oh = g - i * p.PHI; ow = w0 * kTW + (j & 7); n = n0 + i;
      in = i < p.NB && oh < p.TH;
      oh += h0;
    }
    return in && oh < p.OH && ow < p.OW && n < p.N ? (n * p.OH + oh) * p.OW + ow : -1;
  };

  // Pipeline positions; they run on through the passes.
  int sx = 0, sw = 0;                 // stage of the activation ring / weight ring
  uint32_t px = 0, pw = 0;            // parity of the current lap of either ring
  int sp = 0;                         // partial sums so far
  int trades = 0;                     // blocks given and taken (stacked tiles)
  int x_loads = 0, w_loads = 0;
  bool ok = true;
  // Pass 0: scale 16.  If it saw an infinity, pass 1 repeats it looking for the largest FINITE
  // activation.  If the largest one lies outside FP16's window, a pass of two bands follows, and if that
  // saw an activation too small for its lower band (22 bits down to 2^-33 of the largest) one of three.
  // (Always three, and each element's band worked out from its exponent: 128->256 3x3 s2 at 104x104
  // batch 16, all activations 1e-5, 574 us; 356 now.  64->64 3x3 at 56x56 batch 16 84 and 63,
  // 512->512 1x1 at 14x14 batch 16 58.7 and 42.7.)
  bool first = true;
  int bands = 1;
  int emax = 0;                       // exponent of the largest activation (banded passes)
  uint32_t total_at = 0;              // d > 1: a summing warp's columns of its sums
  float total_scale = 1.f;            // d > 1: what takes a summing lane's sums to the output's scale
  // lower end of band b: 2^(emax - 15 - 16 b), zero below the normal numbers
  auto band_end = [&](int b) { const int e = emax + 1 - kBandBits * (b + 1); return e < -126 ? 0.f : pow2f(e); };
  for (;;) {
    const bool banded = bands > 1;
    auto band_exp = [&](int b) { return banded ? min(127, 14 - emax + kBandBits * b) : 4; };  // scale of band b: 2^that
    if (warp == 0) {
      // ---- loads: two independent cursors (patches, weight images) polled in turn ----
      if (lane == 0) {
        const uint32_t box_bytes = (uint32_t)p.box_rows * 128u;
        int xt = tile0, xb = 0, xc = chunk0, xr = 0, xq = 0, oc_, w0, h0, n0;
        int wt = tile0, wb = 0, wc = chunk0, wpr = 0, wpq = 0, wr = 0, wq = 0;
        bool x_left = xt < p.total_tiles && iters > 0, w_left = x_left;
        if (x_left) decode(xt, oc_, w0, h0, n0);
        const __half *wsrc = p.w_tiles + (size_t)(wt - quot(wt, p.by_oc_tiles) * p.oc_tiles) * p.n_chunks * taps * (kWBytes / 2);
        uint32_t idle = 0;
        const uint32_t limit = (uint32_t)abort_flag[1];
        auto load_weights = [&]() {  // the next K step's image
          mbar_expect_tx(bar_wfull(sw), (uint32_t)kWBytes);
          bulk_load(smem_u32(wbase + (size_t)sw * kWBytes), wsrc + ((size_t)wc * taps + wr * p.KS + wq) * (kWBytes / 2), (uint32_t)kWBytes, bar_wfull(sw));
          ++w_loads;
          if (++sw == p.n_w) { sw = 0; pw ^= 1u; }
          if ((wq += p.S) >= p.KS) {
            if ((wr += p.S) >= p.KS) {
              if (++wpq == phases) {
                wpq = 0;
                if (++wpr == phases) {
                  wpr = 0;
                  if (++wc == chunk1) {
                    wc = chunk0;
                    if (++wb == bands) {
                      wb = 0;
                      wt += tile_step;
                      w_left = wt < p.total_tiles;
                      wsrc = p.w_tiles + (size_t)(wt - quot(wt, p.by_oc_tiles) * p.oc_tiles) * p.n_chunks * taps * (kWBytes / 2);
                    }
                  }
                }
              }
              wr = wpr;
            }
            wq = wpq;
          }
        };
        if (first && w_loads == 0) {  // the ring is empty: filled while the launch before this one drains
          while (w_left && w_loads < p.n_w) load_weights();
          grid_wait();
        }
        while (x_left || w_left) {
          bool moved = false;
          if (x_left && mbar_test(bar_xempty(sx), px ^ 1u)) {
            moved = true;
            if (x_loads++ != 0 || !p.withhold_first_load) {  // (test: that patch never arrives, its readers give up)
              const uint32_t dst = smem_u32(xbase + (size_t)sx * p.x_stage_bytes);
              mbar_expect_tx(bar_xfull(sx), box_bytes);
              if (p.mode == kLinear)
                tma_load_4d(dst, &map_x, bar_xfull(sx), xc * KC, w0 * p.npx, 0, 0);
              else if (p.mode == kFlat)  // whole padded rows, from the row of the tile's first position
                tma_load_4d(dst, &map_x, bar_xfull(sx), xc * KC, xq - p.P, quot(w0 * p.npx, p.by_PW) * p.S + xr - p.P, n0);
              else
                tma_load_4d(dst, &map_x, bar_xfull(sx), xc * KC, w0 * kTW * p.S + xq - p.P, h0 * p.S + xr - p.P, n0);
            }
            if (++sx == p.n_x) { sx = 0; px ^= 1u; }
            if (++xq == phases) {
              xq = 0;
              if (++xr == phases) {
                xr = 0;
                if (++xc == chunk1) {
                  xc = chunk0;
                  if (++xb == bands) {
                    xb = 0;
                    xt += tile_step;
                    x_left = xt < p.total_tiles;
                    if (x_left) decode(xt, oc_, w0, h0, n0);
                  }
                }
              }
            }
          }
          if (w_left && mbar_test(bar_wempty(sw), pw ^ 1u)) {
            moved = true;
            load_weights();
          }
          if (moved) { idle = 0; continue; }
          if ((++idle & 31) == 0) {
            if (*abort_flag) { ok = false; break; }
            if (idle >= limit) { *abort_flag = 1; ok = false; break; }
            __nanosleep(20);
          }
        }
      }
    } else if (warp == 1) {
      // ---- MMA issue (converged warp, one elected lane, so that descriptors stay in uniform
      //      registers): per K step one wait, 6 (4) MMAs, one commit ----
      // A K step of the smallest tiles takes the tensor core 200 clocks, about what this warp needs
      // to wait, issue and commit, so the loop is kept short: no early exits (a wait that gave up
      // raises the abort flag, later waits then return at once and the loop runs dry), 3x3 taps
      // unrolled, ring positions counted along.
      const uint32_t idesc = (1u << 4) | ((uint32_t)(p.npx >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
      const uint32_t sbo_x = (uint32_t)(p.mode == kGrid ? p.PW * 128 : 1024);
      const uint64_t dx0 = smem_desc(smem_u32(xbase), sbo_x, 2), dw0 = smem_desc(smem_u32(wbase), STACK ? 512 : 1024, STACK ? 4 : 2);
      const uint32_t dx_hi = (uint32_t)(dx0 >> 32), dw_hi = (uint32_t)(dw0 >> 32);
      const uint32_t x_step = (uint32_t)(p.x_stage_bytes >> 4), row_step = (uint32_t)(p.PW * 8);
      auto wait = [&](uint32_t bar, uint32_t parity) {
        if (!mbar_try_wait(bar, parity)) mbar_wait(bar, parity, abort_flag);
        __syncwarp();
      };
      int k = 0;                  // K step of the band
      auto step = [&](uint32_t xd, bool patch_end) {
        const bool fresh = (k & (p.super - 1)) == 0;
        if (fresh) wait(bar_pempty(sp & 1), ((sp >> 1) & 1) ^ 1);  // first step of a partial sum: its accumulator has been drained
        wait(bar_wfull(sw), pw);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_d = tmem_base + (uint32_t)((sp & 1) * NMAX);
        const uint32_t wd = (uint32_t)dw0 + (uint32_t)(sw * (kWBytes >> 4));
        ++k;
        const bool super_end = k == iters || (k & (p.super - 1)) == 0;
        if (elect_one()) {
          // K slices of 16 channels are 32 bytes = 2 in the address field; x_lo (w_lo) lies 64 bytes after x_hi (w_hi)
          if (STACK) {
            umma_f16_ss(tmem_d, wd, dw_hi, xd, dx_hi, idesc, fresh ? 0u : 1u);
            umma_f16_ss(tmem_d, wd, dw_hi, xd + 4, dx_hi, idesc, 1u);
            umma_f16_ss(tmem_d, wd + 2, dw_hi, xd + 2, dx_hi, idesc, 1u);
            umma_f16_ss(tmem_d, wd + 2, dw_hi, xd + 6, dx_hi, idesc, 1u);
          } else {
            umma_f16_ss(tmem_d, wd, dw_hi, xd, dx_hi, idesc, fresh ? 0u : 1u);
            umma_f16_ss(tmem_d, wd, dw_hi, xd + 4, dx_hi, idesc, 1u);
            umma_f16_ss(tmem_d, wd + 4, dw_hi, xd, dx_hi, idesc, 1u);
            umma_f16_ss(tmem_d, wd + 2, dw_hi, xd + 2, dx_hi, idesc, 1u);
            umma_f16_ss(tmem_d, wd + 2, dw_hi, xd + 6, dx_hi, idesc, 1u);
            umma_f16_ss(tmem_d, wd + 6, dw_hi, xd + 2, dx_hi, idesc, 1u);
          }
          umma_commit(bar_wempty(sw));
          if (super_end) umma_commit(bar_pfull(sp & 1));
          if (patch_end) umma_commit(bar_xempty(sx));
        }
        __syncwarp();
        if (super_end) ++sp;
        if (++sw == p.n_w) { sw = 0; pw ^= 1u; }
      };
      for (int t = tile0; t < p.total_tiles; t += tile_step) {
        uint32_t td0 = (uint32_t)dx0;  // kFlat: the tile's first position lies some columns into its first padded row
        if (p.mode == kFlat) {
          int oc0, w0, h0, n0;
          decode(t, oc0, w0, h0, n0);
          td0 += (uint32_t)((w0 * p.npx - quot(w0 * p.npx, p.by_PW) * p.PW) * 8);
        }
        for (int b = 0; b < bands; ++b) {
          k = 0;
          for (int u = (chunk1 - chunk0) * phases * phases, ph = 0; u > 0; --u) {
            wait(bar_xconv(sx), px);
            const uint32_t xd = td0 + (uint32_t)sx * x_step;
            if (p.KS == 3 && p.S == 1) {
#pragma unroll
              for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int q = 0; q < 3; ++q) step(xd + (uint32_t)r * row_step + 8u * q, r == 2 && q == 2);
            } else {
              const int pr = ph / phases, pq = ph - pr * phases;
              if (++ph == phases * phases) ph = 0;
              uint32_t xrow = xd;
              for (int r = pr; r < p.KS; r += p.S, xrow += row_step) {
                uint32_t xt = xrow;
                for (int q = pq; q < p.KS; q += p.S, xt += 8) step(xt, r + p.S >= p.KS && q + p.S >= p.KS);
              }
            }
            if (++sx == p.n_x) { sx = 0; px ^= 1u; }
          }
        }
      }
    } else if (warp < kFirstSum) {
      // ---- converters: a landed patch, in place, one row per thread: the 16-byte pieces of row r
      //      sit at piece ^ (r & 7) before and after, so the eight lanes of a quarter-warp touch
      //      eight different bank groups ----
      const int ct = (warp - 2) * 32 + lane;
      // bits of the largest |activation|; banded passes: 2 * bits - 1 of the smallest one, zeros last
      unsigned seen = banded ? ~0u : 0u;
      auto note = [&](float a) { seen = __float_as_uint(fmaxf(__uint_as_float(seen), a)); };
      for (int t = tile0; t < p.total_tiles && ok; t += tile_step)
        for (int b = bands - 1; b >= 0 && ok; --b) {
          const float scale = pow2f(band_exp(b));
          const float band_lo = b == bands - 1 ? 0.f : band_end(b), band_hi = band_end(b - 1);  // (infinities and NaN are in the upper band)
          for (int u = (chunk1 - chunk0) * phases * phases; u > 0; --u) {
            if (!(ok = mbar_wait_warp(bar_xfull(sx), px, abort_flag))) break;
            unsigned char *stage = xbase + (size_t)sx * p.x_stage_bytes;
            for (int row = ct; row < p.box_rows; row += 32 * kConv) {
              float4 *rp = reinterpret_cast<float4 *>(stage + (size_t)row * 128);
              if (first)
                convert_row(rp, row & 7, [](float x) { return kXScale * x; }, [&](const float4 &v) {
                  note(fmaxf(fabsf(v.x), fabsf(v.y)));
                  note(fmaxf(fabsf(v.z), fabsf(v.w)));
                });
              else
                seen = convert_row_again(smem_u32(rp), row & 7, scale, band_lo, band_hi, seen, banded ? b : -1);
            }
            // the writes above go through the generic proxy, the MMAs read through the async proxy
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_xconv(sx));
            if (++sx == p.n_x) { sx = 0; px ^= 1u; }
          }
        }
      unsigned m = seen;
      if (banded) m = band_end(1) > 0.f && seen < 2u * __float_as_uint(band_end(1)) - 1u;  // (a third band would hold it)
      for (int s = 16; s; s >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, s));
      if (lane == 0) atomicMax(seen_slot, m);
    } else {
      // ---- summing warps: partials -> running sums -> output.  A warp may touch the TMEM lanes of
      //      its quarter; two warps share a quarter and take half of the pixels each.  (After a
      //      wait that gave up this role, too, runs dry: its warps meet at barriers.) ----
      const int me = warp - kFirstSum, quarter = me & 3, half = me >> 2;
      const int hc = ((p.npx >> 4) + 1) / 2 * 16;                 // pixels of the first half
      const int j0 = half * hc, ncols = half ? p.npx - hc : hc;   // this warp's pixels
      const int ocl = STACK ? (quarter & 1) * 32 + lane : quarter * 32 + lane;  // channel inside the tile
      int4 *gtab = gtabs + me * (NC / 8);
      float *blocks = reinterpret_cast<float *>(exch) + me * 1024;             // two blocks of 16 pixels x 32 channels
      float *give = reinterpret_cast<float *>(exch) + kSumWarps * 1024 + me * 1024;  // stacked tiles
      const float *take = reinterpret_cast<const float *>(exch) + kSumWarps * 1024 + (me ^ 2) * 1024;
      int nblk = 0;
      const float unscale = banded ? pow2f(4 - band_exp(0)) : 1.f;
      for (int t = tile0; t < p.total_tiles; t += tile_step) {
        int oc0, w0, h0, n0;
        decode(t, oc0, w0, h0, n0);
        __syncwarp();
        if (p.d == 1 && lane < NC / 8) {
          // where this warp's pixel group `lane` goes: {x, row, image} of a box of 8 pixels in the
          // output tensor (what lies past the tensor is dropped), or pixel by pixel
          int4 e = make_int4(0, 0, n0, 0);  // w: 0 nowhere, 1 a box, 2 pixel by pixel
          const int j = j0 + 8 * lane;
          if (8 * lane < ncols) {
            if (p.mode == kLinear) {
              e.x = w0 * p.npx + j;
              e.w = e.x < p.total_pixels ? 1 : 0;
            } else if (p.mode == kFlat) {
              const int pos = w0 * p.npx + j;
              e.y = quot(pos, p.by_PW); e.x = pos - e.y * p.PW;
              e.w = e.y >= p.OH ? 0 : e.x + 8 > p.PW ? 2 : e.x < p.OW ? 1 : 0;
            } else {
              const int g = j >> 3, i = p.NB > 1 ? quot(g, p.by_PHI) : 0;
              e.x = w0 * kTW; e.y = g - i * p.PHI; e.z = n0 + i;
              e.w = i < p.NB && e.y < p.TH && h0 + e.y < p.OH && e.z < p.N ? 1 : 0;
              e.y += h0;
            }
            if (e.w == 1 && !p.tma_store) e.w = 2;
          }
          gtab[lane] = e;
        }
        __syncwarp();
        // Sum the partials in registers; the total goes back into the last partial's columns of
        // tensor memory, from where a short loop takes it on (16 pixels at a time, the same code
        // every time: 128 registers can only be walked by unrolled code, which ran at the rate of
        // the instruction fetches -- 9000 clocks per tile).  An item of one partial is taken as it is.
        const int partials = supers * bands;
        auto partial = [&]() {  // this warp's first column of the next partial, once the tensor core is done with it
          if (!mbar_try_wait(bar_pfull(sp & 1), (sp >> 1) & 1)) mbar_wait(bar_pfull(sp & 1), (sp >> 1) & 1, abort_flag);
          __syncwarp();
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          return tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((sp & 1) * NMAX + j0);
        };
        uint32_t ttotal;
        if (partials > 1) {
          float acc[NC];
#pragma unroll
          for (int j = 0; j < NC; ++j) acc[j] = 0.f;
          int left = supers, band = bands - 1;
#pragma unroll 1
          for (int i = 1; i < partials; ++i, ++sp) {
            const uint32_t taddr = partial();
#pragma unroll
            for (int c0 = 0; c0 < NC; c0 += 16) {
              if (c0 < ncols) {
                uint32_t v[16];
                tmem_ld16(taddr + c0, v);
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c0 + j] += __uint_as_float(v[j]);
              }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_pempty(sp & 1));  // the tensor core may overwrite the partial
            if (--left == 0) {  // from this band's scale to the next larger one's
              const float f = pow2f(band_exp(band - 1) - band_exp(band));
              left = supers; --band;
#pragma unroll
              for (int j = 0; j < NC; ++j) acc[j] *= f;
            }
          }
          ttotal = partial();
#pragma unroll
          for (int c0 = 0; c0 < NC; c0 += 16) {
            if (c0 < ncols) {
              uint32_t v[16];
              tmem_ld16(ttotal + c0, v);
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(acc[c0 + j] + __uint_as_float(v[j]));
              tmem_st16(ttotal + c0, v);
            }
          }
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        } else {
          ttotal = partial();
        }
        ++sp;
        // The sums leave by one multiplication by 2^-sh[oc] / 16 times the banded pass's own factor, exact
        // as powers of two.  Each factor alone can take a sum (up to 2^30) out of FP32's range though the
        // result is inside it (|x| of 2^112 and weights of 0.05), and where both are tiny so can their
        // product: there the sums take the banded pass's factor first, where they lie.
        const int oc = oc0 + ocl;
        const float channel_scale = oc < p.OC ? p.out_scale[oc] : 0.f;
        float sc = channel_scale * unscale;
        if (banded) {
          const bool apart = channel_scale != 0.f && !(sc >= 1.17549435e-38f && sc <= 3.402823466e38f);
          if (__any_sync(0xffffffffu, apart)) {
            scale_columns(ttotal, ncols, apart ? unscale : 1.f);
            if (apart) sc = channel_scale;
          }
        }
        if (p.d > 1) {
          total_at = ttotal;  // a slice of a tile: its sums stay in tensor memory until the cluster meets
          total_scale = sc;
        } else {
          // Store: a thread holds one channel of many pixels, an 8-pixel group of a warp is a box of
          // 32 channels x 8 pixels of the output.  16 pixels at a time go into a staging block (one
          // conflict-free 4-byte store per value), which TMA stores carry on from there while the
          // warp stages the next block.
          const int ocw = oc - lane;  // first channel of the warp
          auto put16 = [&](int c0, const float (&v)[16]) {  // pixels c0 .. c0 + 15 of this warp
            float *blk = blocks + (nblk & 1) * 512;
            ++nblk;
            if (lane < 2) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");  // the stores of the block before last have read it
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 16; ++j) blk[j * 32 + lane] = p.relu ? fmaxf(v[j] * sc, 0.f) : v[j] * sc;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            const int4 mine = gtab[(c0 >> 3) + (lane & 1)];  // (even lanes: first group, odd lanes: second)
            __syncwarp();
            if (lane < 2) {
              if (mine.w == 1 && ocw < p.OC)
                asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
                             ::"l"(&map_out), "r"(smem_u32(blk + lane * 256)), "r"(ocw), "r"(mine.x), "r"(mine.y), "r"(mine.z) : "memory");
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
            if (__any_sync(0xffffffffu, mine.w == 2)) {
              const int wa = __shfl_sync(0xffffffffu, mine.w, 0), wb = __shfl_sync(0xffffffffu, mine.w, 1);
#pragma unroll 1
              for (int j = wa == 2 ? 0 : 8; j < (wb == 2 ? 16 : 8); ++j) {
                const int pix = pixel_of(j0 + c0 + j, w0, h0, n0);
                if (pix >= 0 && oc < p.OC) p.out[(size_t)pix * p.OC + oc] = blk[j * 32 + lane];
              }
            }
          };
          if (STACK) {
            // Lanes 64..127 hold the w_lo halves of the channels of lanes 0..63.  The two warps of a
            // channel group and half give each other 16 pixels at a time through shared memory -- the
            // w_lo warp from the first half of the pixels, the other one from the second -- and store
            // the rest.  Two blocks in turn: one barrier per round.
            const int split = ((ncols >> 4) + 1) / 2 * 16;
            const int out0 = quarter >= 2 ? 0 : split, nout = quarter >= 2 ? split : ncols - split;  // pixels given away
            const int in0 = quarter >= 2 ? split : 0, nin = ncols - nout;                            // pixels kept
#pragma unroll 1
            for (int c = 0; c < split; c += 16) {
              uint32_t v[16];
              const int slot = (trades++ & 1) * 512 + lane;
              if (c < nout) {
                tmem_ld16(ttotal + out0 + c, v);
#pragma unroll
                for (int j = 0; j < 16; ++j) give[slot + j * 32] = __uint_as_float(v[j]);
              }
              asm volatile("bar.sync %0, 64;" ::"r"(1 + half * 2 + (quarter & 1)) : "memory");
              if (c < nin) {
                tmem_ld16(ttotal + in0 + c, v);
                float y[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) y[e] = __uint_as_float(v[e]) + take[slot + e * 32];
                put16(in0 + c, y);
              }
            }
          } else {
#pragma unroll 1
            for (int c0 = 0; c0 < ncols; c0 += 16) {
              uint32_t v[16];
              tmem_ld16(ttotal + c0, v);
              float y[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) y[j] = __uint_as_float(v[j]);
              put16(c0, y);
            }
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_pempty((sp - 1) & 1));
      }
      if (lane < 2) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // this warp's stores are complete
    }
    // ---- end of a pass: does this CTA's largest activation ask for another one? ----
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned m = *reinterpret_cast<volatile unsigned *>(seen_slot);
    const bool in_window = m < 0x45000000u && (m == 0u || m >= 0x3B800000u);
    if (*abort_flag != 0 || bands == 3 || (bands == 2 ? m == 0u : in_window)) break;
    if (bands == 2) {
      bands = 3;
    } else if (m < 0x7F800000u) {
      bands = 2;
      emax = (int)(m >> 23) - 127;
    }
    first = false;
    __syncthreads();
    if (tid == 0) *seen_slot = 0u;
    __syncthreads();
  }

  if (*abort_flag) {  // what this CTA has in flight must land before it leaves
    if (tid == 0) {
      for (int v = max(x_loads - p.n_x, p.withhold_first_load ? 1 : 0); v < x_loads; ++v) mbar_drain(bar_xfull(v % p.n_x), (uint32_t)(v / p.n_x) & 1u);
      for (int v = max(w_loads - p.n_w, 0); v < w_loads; ++v) mbar_drain(bar_wfull(v % p.n_w), (uint32_t)(v / p.n_w) & 1u);
    }
    if (warp == 1) {
      if (elect_one()) umma_commit(bar_drain());
      __syncwarp();
      mbar_drain(bar_drain(), 0);
    }
    if (tid == 0) atomicExch(p.error_flag, 1);
  }
  if (p.d > 1) {
    // The slices of a tile meet.  Each CTA owns a share of the tile's pixels; once every ring of the
    // cluster is idle, the summing warps write their sums of a pixel, at the output's scale, into its owner's
    // shared memory (one row of 128 accumulator lanes per slice and pixel), and the owner adds the rows up in
    // slice order and stores the result.  The code is small on purpose: it runs once, at the rate of its instruction
    // fetches.  (Sums fetched from the other CTAs, four pixels per warp unrolled, and a barrier behind
    // the stores took 6000 to 14000 clocks whatever the amount of data.)
    const int per = share_pixels(p.npx, p.d);
    cluster_sync_all();
    if (warp >= kFirstSum && !*abort_flag) {
      const int me = warp - kFirstSum, quarter = me & 3, half = me >> 2;
      const int hc = ((p.npx >> 4) + 1) / 2 * 16, j0 = half * hc, ncols = half ? p.npx - hc : hc;
      const uint32_t row = smem_u32(xbase) + (uint32_t)(quarter * 32 + lane) * 4u;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
      for (int c0 = 0; c0 < ncols; c0 += 16) {
        const int owner = (j0 + c0) / per;
        const uint32_t dst = cluster_addr(row + (uint32_t)((rank * per + j0 + c0 - owner * per) * BM) * 4u, (uint32_t)owner);
        uint32_t v[16];
        tmem_ld16(total_at + c0, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) st_cluster(dst + (uint32_t)(j * BM) * 4u, __uint_as_float(v[j]) * total_scale);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncwarp();
    cluster_sync_all();  // (all rows have arrived; nothing reaches into another CTA after this)
    int oc0, w0, h0, n0;
    decode(tile0, oc0, w0, h0, n0);
    constexpr int kPix = STACK ? 2 : 1;                // pixels of a warp at a time; a lane adds up four channels
    const int l4 = 4 * (STACK ? lane & 15 : lane), oc = oc0 + l4;
    const bool vec = (p.OC & 3) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
    const float4 *rows = reinterpret_cast<const float4 *>(xbase) + (l4 >> 2);
    const int jend = *abort_flag ? 0 : min(per, p.npx - rank * per);
#pragma unroll 1
    for (int j = warp * kPix + (STACK ? lane >> 4 : 0); j < jend; j += kThreads / 32 * kPix) {
      float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
      for (int s = 0; s < p.d; ++s) {
        float4 u = rows[(s * per + j) * (BM / 4)];
        if (STACK) {
          const float4 l = rows[(s * per + j) * (BM / 4) + 16];
          u.x += l.x; u.y += l.y; u.z += l.z; u.w += l.w;
        }
        y.x += u.x; y.y += u.y; y.z += u.z; y.w += u.w;
      }
      const int pix = pixel_of(rank * per + j, w0, h0, n0);
      if (pix < 0 || oc >= p.OC) continue;
      float v[4] = {y.x, y.y, y.z, y.w};
      if (p.relu) {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = fmaxf(v[i], 0.f);
      }
      float *o = p.out + (size_t)pix * p.OC + oc;
      if (vec) *reinterpret_cast<float4 *>(o) = make_float4(v[0], v[1], v[2], v[3]);
      else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (oc + i < p.OC) o[i] = v[i];
      }
    }
  }
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
}

// Per output channel: the power of two that brings the channel's largest |w| into [2^12, 2^13)
// (1 for an all-zero channel), and its inverse divided by the activation scale.
__global__ void tc16_scales_kernel(const float *__restrict__ w, int per_oc, float *__restrict__ w_scale, float *__restrict__ out_scale) {
  const float *row = w + (size_t)blockIdx.x * per_oc;
  unsigned m = 0;
  for (int i = threadIdx.x; i < per_oc; i += blockDim.x) {
    const unsigned b = __float_as_uint(row[i]) & 0x7FFFFFFFu;
    if (b < 0x7F800000u) m = max(m, b);
  }
  __shared__ unsigned red[32];
  for (int d = 16; d; d >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, d));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < (int)(blockDim.x >> 5); ++i) m = max(m, red[i]);
    int sh = 0;
    if (m) {
      int e;
      frexpf(__uint_as_float(m), &e);  // |w|max = f * 2^e, f in [0.5, 1)
      sh = min(100, max(-100, 13 - e));
    }
    w_scale[blockIdx.x] = ldexpf(1.f, sh);
    out_scale[blockIdx.x] = ldexpf(1.f, -sh) / kXScale;
  }
}

typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                             const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                             CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn get_encode() {
  static EncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess) fn = (EncodeFn)p;
  });
  return fn;
}

// How one conv shape runs: tile geometry, K slices, rings.
struct Geometry {
  int mode = -1, npx = 0, PW = 0, PHI = 0, TH = 1, NB = 1;
  int tiles_w = 1, tiles_h = 1, tiles_n = 1;
  int box_w = 1, box_h = 1, box_n = 1, reach = 0;  // patch load; furthest row a window touches
  int d = 1, nmax = 128, n_x = 2, n_w = 3, x_stage = 0;
  size_t smem = 0;
  // Estimated clocks.  `cost` leaves out what loads cost and comes out a quarter below `rank`; the list kernel's
  // model it is compared with comes out low as well, and with `rank` in its place that comparison chose worse
  // (untuned layers, 356 of them: 1.6 % above the faster kernel on average, 3.5 % with `rank`).
  double cost = 0.;  // to compare with the list kernel's model
  double rank = 0.;  // to compare geometries
};

struct Tc16State {
  __half *d_tiles = nullptr;
  int *d_error = nullptr;
  float *d_out_scale = nullptr;  // per output channel
  int n_chunks = 0, oc_tiles = 1, sms = 0;
  bool stack = false;            // at most 64 output channels: {w_hi, w_lo} stacked on the M side
  // Launch set-ups (tensor map, tile plan, grid), one per (input pointer, conv shape) seen lately.
  struct Setup {
    bool valid = false;
    const float *in = nullptr;
    const float *out = nullptr;
    ConvShape shape{};
    CUtensorMap map_x, map_out;
    Tc16Params params{};
    unsigned grid = 0;
    int nmax = 128;
    size_t smem = 0;
  };
  static constexpr int kSetups = 8;
  std::mutex mutex;
  Setup setups[kSetups];
  int next_setup = 0;
  Geometry last_geo;             // geometry of the last shape planned (independent of the pointers)
  ConvShape last_shape{};
};

constexpr size_t kSmemBudget = 227 * 1024;

bool same_conv(const ConvShape &a, const ConvShape &b) {
  return a.N == b.N && a.H == b.H && a.W == b.W && a.S == b.S && a.P == b.P;
}

// Rings and estimated time of a geometry whose tile is settled; false if it does not fit.
bool finish_geometry(const Tc16State &t, const ConvShape &s, Geometry *g) {
  const int taps = s.KS * s.KS, phases = std::min(s.S, s.KS);
  const size_t wb = t.stack ? 8192 : 16384;
  const int box_rows = g->box_w * g->box_h * g->box_n;
  if (g->box_w * s.S > 256 || g->box_h * s.S > 256 || g->box_n > 256) return false;
  g->nmax = g->npx > 128 ? 256 : 128;
  g->x_stage = (std::max(g->reach, box_rows) * 128 + 1023) / 1024 * 1024;
  const size_t fixed = 1024 + stage_bytes(t.stack) + kNumBars * 8 + kSumWarps * (g->nmax / 16) * 16 + 64;
  auto fits = [&](int nx, int nw) { return fixed + (size_t)nx * g->x_stage + nw * wb <= kSmemBudget; };
  if (!fits(2, 3)) return false;
  // a patch feeds taps / phases^2 K steps: filters larger than 1x1 need few patches and many weight
  // images in flight, 1x1 filters one of each per K step
  const int steps = std::max(1, taps / (phases * phases));
  const int x_want = steps >= 4 ? 3 : kXStagesMax;
  g->n_x = 2; g->n_w = 3;
  for (bool grew = true; grew;) {
    grew = false;
    if (g->n_x < std::min(x_want, 3) && fits(g->n_x + 1, g->n_w)) { ++g->n_x; grew = true; }
    if (g->n_w < kWStagesMax && fits(g->n_x, g->n_w + 1)) { ++g->n_w; grew = true; }
    if (g->n_x < x_want && fits(g->n_x + 1, g->n_w)) { ++g->n_x; grew = true; }
  }
  // (more than half of an SM's: the CTAs of a launch that is placed while another one drains must
  // not be doubled up on the SMs that are free first)
  g->smem = std::max(fixed + (size_t)g->n_x * g->x_stage + g->n_w * wb, (size_t)116 * 1024);
  if (g->d > 1 && (size_t)g->d * share_pixels(g->npx, g->d) * BM * 4 > (size_t)g->n_x * g->x_stage + g->n_w * wb) return false;  // (the sums of a slice)
  // clocks per K step: the MMAs themselves, the shared-memory pipe (MMA operands, weight copy,
  // patch landing, read and written by the conversion), the conversion, the issuing warp
  const int nm = t.stack ? 4 : 6, conv = g->nmax == 256 ? 2 : 6;
  const double operand = 4096. + 32. * g->npx;
  const double mma = nm * std::max(0.52 * g->npx, operand / 128.);
  const double pipe = (nm * operand + wb + 384. * box_rows / steps) / 128.;
  const double cvt = std::ceil(box_rows / (32. * conv)) * 420. / steps;
  const double step = std::max(std::max(mma, pipe), std::max(cvt, 330.));
  const double k_steps = (double)taps * ((t.n_chunks + g->d - 1) / g->d);
  const double tiles = (double)g->tiles_w * g->tiles_h * g->tiles_n * t.oc_tiles;
  // (clusters of d CTAs live inside a GPC: on the 148-SM part 148 CTAs in pairs, 132 in fours, 120 in eights)
  const double slots = g->d <= 2 ? t.sms : g->d * std::floor(t.sms * (g->d == 4 ? 0.225 : 0.1015));
  const double waves = std::ceil(tiles * g->d / slots);
  // (channel counts TMA stores do not take leave value by value: 32->17 3x3 at 112x112 batch 4, 26.9 us against
  // 14.7 with 16 channels; with 12 clocks a pixel there, too, it was chosen before the list kernel's 15.4)
  const double item = std::max(k_steps * step, ((s.OC & 3) == 0 || g->d > 1 ? 12. : 33.) * g->npx) + 400.;
  g->cost = waves * item + 5000. + 10. * g->npx + 0.3 * box_rows * 10. + (g->d > 1 ? 2500. + 8. * g->npx + (waves - 1.) * 5000. : 0.);
  // The geometries among themselves.  Measured on 26 layers, batch 1 to 16: loads reach an SM at about 30
  // bytes per clock, weights (which many CTAs ask for at once) slower than patches -- 1x1 96 pixels
  // 920 to 1160 clocks per K step (28 KB), 3x3 96 pixels 640 (18 KB), 176 pixels 1450 (38 KB); a K step
  // of the smallest tiles takes 450; 6000 clocks pass before the first MMA; an epilogue takes 2000 clocks
  // (32 pixels) to 4400 (176); a cluster meets in 3400 (16 pixels), 5300 (96), 7000 (112), 13000 (224).
  // Without the load term small tiles in many CTAs looked cheap: 1x1 1024->1024 at 7x7 batch 1 took 128
  // CTAs of 16 pixels, 11.8 us; 64 of 64 pixels take 9.6; 256->64 at 56x56 batch 16 128 pixels, 22.0,
  // against 176, 19.8; 3x3 64->64 at 56x56 batch 1 10.1 against 9.2.
  const double loads = wb / 24. + 128. * box_rows / steps / 40.;
  const double slow = std::max(std::max(step, 450.), loads);
  const double meet = g->d > 1 ? 2000. + 45. * g->npx : 1000. + 22. * g->npx;
  g->rank = waves * (std::max(k_steps * slow, 12. * g->npx) + 400.) + 6000. + 3. * box_rows + meet +
            (g->d > 1 ? (waves - 1.) * (6000. + meet) : 0.);
  return true;
}

// The cheapest geometry by that estimate.
bool plan_geometry(const Tc16State &t, const ConvShape &s, Geometry *best) {
  const int amax = (s.KS - 1) / s.S;
  bool found = false;
  auto consider = [&](Geometry g) {
    for (int d = 1; d <= 8 && d <= t.n_chunks; d *= 2) {
      g.d = d;
      Geometry c = g;
      if (finish_geometry(t, s, &c) && (!found || c.rank < best->rank)) { *best = c; found = true; }
    }
  };
  const long long pixels = (long long)s.N * s.OH * s.OW;
  for (int npx = 16; npx <= 256; npx += 16) {
    Geometry g;
    g.npx = npx;
    if (s.KS == 1 && s.S == 1 && s.P == 0) {
      g.mode = kLinear;
      g.PW = kTW; g.PHI = 1;
      g.tiles_w = (int)((pixels + npx - 1) / npx);
      g.box_w = npx; g.reach = npx;
      consider(g);
      continue;
    }
    // whole padded rows
    if ((long long)s.OH * (s.OW + amax) >= (1ll << 31) - 1024) continue;
    g.mode = kFlat;
    g.PW = s.OW + amax;
    g.TH = s.OH;
    g.PHI = (g.PW - 1 + npx - 1) / g.PW + 1 + amax;
    g.tiles_w = ((s.OH - 1) * g.PW + s.OW + npx - 1) / npx;
    g.tiles_n = s.N;
    g.box_w = g.PW; g.box_h = g.PHI;
    g.reach = g.PW - 1 + npx + amax * g.PW + amax;
    consider(g);
  }
  if (s.KS == 1 && s.S == 1 && s.P == 0) return found;
  for (int cuts = (s.OH + 31) / 32, last = 0; cuts <= s.OH; ++cuts) {
    const int TH = (s.OH + cuts - 1) / cuts;
    if (TH == last) continue;
    last = TH;
    for (int NB = 1; NB <= s.N; ++NB) {
      if (NB > 1 && (TH != s.OH || (NB - 1) * (TH + amax) + TH > 32)) break;
      Geometry g;
      g.mode = kGrid;
      g.TH = TH; g.NB = NB;
      g.PW = kTW + amax; g.PHI = TH + amax;
      const int groups = ((NB - 1) * g.PHI + TH + 1) / 2 * 2;
      g.npx = 8 * groups;
      g.tiles_w = (s.OW + kTW - 1) / kTW;
      g.tiles_h = (s.OH + TH - 1) / TH;
      g.tiles_n = (s.N + NB - 1) / NB;
      g.box_w = g.PW; g.box_h = g.PHI; g.box_n = NB;
      g.reach = (groups - 1 + amax) * g.PW + amax + kTW;
      consider(g);
    }
  }
  return found;
}

// K steps the tensor core adds up before the sum is carried on outside: the error of an output, which is
// that of the truncating adds inside a partial, grows with it (relative, against 64 bits, 256 channels and
// more: 7.2e-7 with 8 steps, 4.0e-7 with 4, 2.4e-7 with 2, 1.6e-7 with 1; split TF32, whose K step is 12
// MMAs instead of 6: 5.3e-7 with its 4 steps, 3.1e-7 with 2, 2.0e-7 with 1), and so does the speed: on VGG-19
// at batch 16, 3x3 layers of 128 channels and more, 4 steps cost 1 to 11 % against 8, on 1x1 layers 0 to 4 %,
// 2 steps 4 % more.  The rule keeps every layer at the error of the faster tensor-core kernel there was
// for it before this one, or below:
//   * larger filters than 1x1 at stride 1 with more than 32 channels and more than two waves of 128-pixel
//     tiles: 8, as the split-FP16 kernel had that ran them (with fewer channels or tiles its fixed costs
//     showed and split TF32 was faster: 24->128 at 112x112 batch 4 24.7 us against 26.7, 64->128 41.4 to 35.0);
//   * others: 4, as the split-TF32 kernel that ran them has; 1x1 layers of few tiles, whose K range that
//     kernel cuts into slices added up in FP32, no more steps than a slice has;
//   * stacked filters do a K step in 4 MMAs and carry the same error over twice the steps (8: 4.7e-7).
int partial_steps(const Tc16State &t, const ConvShape &s) {
  const long long pixels = (long long)s.N * s.OH * s.OW, tiles = (pixels + 127) / 128 * t.oc_tiles;
  if (s.KS > 1 && s.S == 1 && t.n_chunks > 1 && tiles > 2ll * t.sms) return 8;
  int steps = 4;
  if (s.KS == 1)
    for (int d = 2; d <= 8 && tiles * d <= t.sms; ++d)
      if (t.n_chunks % d == 0)
        while (steps > 1 && steps > t.n_chunks / d) steps /= 2;
  return t.stack && s.S == 1 ? 2 * steps : steps;
}

// The geometry of a shape, planned once (the caller holds the state's mutex).
const Geometry *geometry_of(Tc16State *t, const ConvShape &s) {
  if (t->last_geo.mode < 0 || !same_conv(t->last_shape, s)) {
    t->last_geo = Geometry{};
    if (!plan_geometry(*t, s, &t->last_geo)) { t->last_geo.mode = -1; return nullptr; }
    t->last_shape = s;
  }
  return &t->last_geo;
}

template <int NMAX, bool STACK>
int launch_instance(const CUtensorMap &map_x, const CUtensorMap &map_out, const Tc16Params &p, unsigned grid, size_t smem, cudaStream_t st) {
  static thread_local bool configured[16] = {false};
  int dev = 0;
  TETRIS_CUDA_TRY(cudaGetDevice(&dev));
  if (dev >= 16 || !configured[dev]) {
    TETRIS_CUDA_TRY(cudaFuncSetAttribute(conv_tc16_kernel<NMAX, STACK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
    if (dev < 16) configured[dev] = true;
  }
  TETRIS_CUDA_TRY(launch_overlapped(conv_tc16_kernel<NMAX, STACK>, dim3(grid), Roles<NMAX>::kThreads, smem, st, (unsigned)p.d, map_x, map_out, p));
  return TETRIS_OK;
}

}  // namespace

void conv_tc16_state_delete(void *state) {
  Tc16State *s = static_cast<Tc16State *>(state);
  if (!s) return;
  device_free(s->d_tiles);
  delete s;
}

// Makes room for the split FP16 weight images and works out the scales (called from filter creation
// and from the file loader; d_dense is the OIHW filter on the device).  Failure here is not fatal
// for the filter: the variant is then reported as unsupported.
int conv_tc16_prepare(tetris_filter *f, const float *d_dense, WeightImages *w) {
  if (f->groups != 1 || (f->in_channel & 3) != 0 || f->in_channel < 8 || f->kernel_size > 7) return TETRIS_OK;
  Tc16State *s = new (std::nothrow) Tc16State();
  if (!s) return TETRIS_OK;
  const int KS = f->kernel_size, taps = KS * KS;
  s->n_chunks = (f->in_channel + KC - 1) / KC;
  s->stack = f->out_channel <= 64;
  s->oc_tiles = (f->out_channel + BM - 1) / BM;
  const size_t tile_bytes = (size_t)taps * s->n_chunks * s->oc_tiles * BM * (s->stack ? 64 : 128);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&s->sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) s->sms = 0;
  // one buffer: images, scales of the outputs and of the weights, error flag
  if (s->sms < 1 || device_alloc((void **)&s->d_tiles, tile_bytes + 2 * f->out_channel * sizeof(float) + sizeof(int)) != cudaSuccess) {
    cudaGetLastError();
    conv_tc16_state_delete(s);
    return TETRIS_OK;
  }
  s->d_out_scale = reinterpret_cast<float *>(reinterpret_cast<char *>(s->d_tiles) + tile_bytes);
  float *d_w_scale = s->d_out_scale + f->out_channel;
  s->d_error = reinterpret_cast<int *>(d_w_scale + f->out_channel);
  cudaMemsetAsync(s->d_error, 0, sizeof(int), 0);
  // per-channel scales: every output channel's largest |w| lands in [2^12, 2^13)
  tc16_scales_kernel<<<f->out_channel, 256>>>(d_dense, f->in_channel * taps, d_w_scale, s->d_out_scale);
  if (cudaGetLastError() != cudaSuccess) {
    conv_tc16_state_delete(s);
    return TETRIS_OK;
  }
  w->tc16 = s->d_tiles;
  w->stack = s->stack ? 1 : 0;
  w->scale = d_w_scale;
  f->tc16_state = s;
  return TETRIS_OK;
}

bool conv_tc16_supported(const tetris_filter *f, const ConvShape &s) {
  if (!f->tc16_state || f->groups != 1) return false;
  if (s.S < 1 || s.S > 4 || s.N < 1 || s.OH < 1 || s.OW < 1) return false;
  // (pixel numbers and image coordinates are 32-bit, and a tile reaches up to 256 of them past the last one)
  constexpr long long kMost = (1ll << 31) - 1024;
  return (long long)s.N * s.OH * s.OW < kMost && s.H + 2ll * s.P < kMost && s.W + 2ll * s.P < kMost;
}

// Estimated clocks of a launch (negative: the shape is not covered).
double conv_tc16_cost(const tetris_filter *f, const ConvShape &s) {
  if (!conv_tc16_supported(f, s)) return -1.;
  Tc16State *t = static_cast<Tc16State *>(f->tc16_state);
  std::lock_guard<std::mutex> lock(t->mutex);
  const Geometry *g = geometry_of(t, s);
  return g ? g->cost : -1.;
}

int launch_conv_tc16(const tetris_filter *f, const float *in, float *out, const ConvShape &s, cudaStream_t st) {
  Tc16State *t = static_cast<Tc16State *>(f->tc16_state);
  if (!conv_tc16_supported(f, s) || (reinterpret_cast<uintptr_t>(in) & 15) != 0) {
    set_error("split-FP16 tensor-core variant covers strides up to 4, in_channel a multiple of 4 (at least 8), 16-byte aligned inputs");
    return TETRIS_ERR_UNSUPPORTED;
  }
  EncodeFn enc = get_encode();
  if (!enc) { set_error("cuTensorMapEncodeTiled is not available from this driver"); return TETRIS_ERR_UNSUPPORTED; }
  CUtensorMap map_x, map_out;
  Tc16Params p;
  unsigned grid = 0;
  int nmax = 128;
  size_t smem = 0;
  {
    std::lock_guard<std::mutex> lock(t->mutex);
    Tc16State::Setup *su = nullptr;
    for (Tc16State::Setup &c : t->setups)
      if (c.valid && c.in == in && c.out == out && same_conv(c.shape, s)) { su = &c; break; }
    if (!su) {
      const Geometry *g = geometry_of(t, s);
      if (!g) { set_error("split-FP16 variant: the activation patches of this layer do not fit shared memory"); return TETRIS_ERR_UNSUPPORTED; }
      su = &t->setups[t->next_setup];
      t->next_setup = (t->next_setup + 1) % Tc16State::kSetups;
      su->valid = false;
      Tc16Params &q = su->params;
      q = Tc16Params{};
      q.N = s.N; q.OH = s.OH; q.OW = s.OW; q.OC = s.OC; q.S = s.S; q.P = s.P; q.KS = s.KS;
      q.mode = g->mode; q.npx = g->npx; q.PW = g->PW; q.PHI = g->PHI; q.TH = g->TH; q.NB = g->NB;
      q.box_rows = g->box_w * g->box_h * g->box_n;
      q.x_stage_bytes = g->x_stage; q.n_x = g->n_x; q.n_w = g->n_w;
      q.tiles_w = g->tiles_w; q.tiles_h = g->tiles_h; q.tiles_n = g->tiles_n; q.oc_tiles = t->oc_tiles;
      q.total_tiles = g->tiles_w * g->tiles_h * g->tiles_n * t->oc_tiles;
      q.by_oc_tiles = fast_div(q.oc_tiles); q.by_tiles_w = fast_div(q.tiles_w); q.by_tiles_h = fast_div(q.tiles_h);
      q.by_PW = fast_div(q.PW); q.by_PHI = fast_div(q.PHI);
      q.n_chunks = t->n_chunks; q.d = g->d;
      q.super = partial_steps(*t, s);
      q.total_pixels = (long long)s.N * s.OH * s.OW;
      q.out_scale = t->d_out_scale; q.error_flag = t->d_error; q.w_tiles = t->d_tiles;
      cuuint64_t dims[4], strides[3];
      cuuint32_t box[4], estr[4] = {1, (cuuint32_t)s.S, (cuuint32_t)s.S, 1};
      if (g->mode == kLinear) {
        dims[0] = (cuuint64_t)s.IC; dims[1] = (cuuint64_t)q.total_pixels; dims[2] = 1; dims[3] = 1;
        strides[0] = (cuuint64_t)s.IC * 4; strides[1] = strides[0] * dims[1]; strides[2] = strides[1];
      } else {
        dims[0] = (cuuint64_t)s.IC; dims[1] = (cuuint64_t)s.W; dims[2] = (cuuint64_t)s.H; dims[3] = (cuuint64_t)s.N;
        strides[0] = (cuuint64_t)s.IC * 4; strides[1] = strides[0] * s.W; strides[2] = strides[1] * s.H;
      }
      // with element strides a box spans S times the pixels it loads
      box[0] = KC; box[1] = (cuuint32_t)(g->box_w * s.S); box[2] = (cuuint32_t)(g->box_h * s.S); box[3] = (cuuint32_t)g->box_n;
      const CUresult r = enc(&su->map_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float *>(in), dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
      if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled failed with code %d", (int)r); return TETRIS_ERR_CUDA; }
      // the output as boxes of 32 channels x 8 pixels
      std::memset(&su->map_out, 0, sizeof(su->map_out));
      q.tma_store = 0;
      if ((s.OC & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
        cuuint64_t odims[4] = {(cuuint64_t)s.OC, (cuuint64_t)s.OW, (cuuint64_t)s.OH, (cuuint64_t)s.N}, ostrides[3];
        if (g->mode == kLinear) { odims[1] = (cuuint64_t)q.total_pixels; odims[2] = odims[3] = 1; }
        ostrides[0] = odims[0] * 4; ostrides[1] = ostrides[0] * odims[1]; ostrides[2] = ostrides[1] * odims[2];
        const cuuint32_t obox[4] = {32, kTW, 1, 1}, oestr[4] = {1, 1, 1, 1};
        if (enc(&su->map_out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, out, odims, ostrides, obox, oestr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS)
          q.tma_store = 1;
      }
      // persistent CTAs, one per SM; a tile cut into K slices takes a cluster of its own
      su->grid = (unsigned)(g->d > 1 ? q.total_tiles * g->d : std::min(q.total_tiles, t->sms));
      su->nmax = g->nmax;
      su->smem = g->smem;
      su->in = in;
      su->out = out;
      su->shape = s;
      su->valid = true;
    }
    map_x = su->map_x;
    map_out = su->map_out;
    p = su->params;
    grid = su->grid;
    nmax = su->nmax;
    smem = su->smem;
  }
  p.out = out;
  p.relu = s.relu;
  p.withhold_first_load = test_injection(&p.spin_limit);
  const int rc = nmax == 256 ? (t->stack ? launch_instance<256, true>(map_x, map_out, p, grid, smem, st) : launch_instance<256, false>(map_x, map_out, p, grid, smem, st))
                             : (t->stack ? launch_instance<128, true>(map_x, map_out, p, grid, smem, st) : launch_instance<128, false>(map_x, map_out, p, grid, smem, st));
  if (rc) return rc;
  count_launch();
  if (p.relu) note_relu_fused();
  return TETRIS_OK;
}

// 0 = no timeout seen so far, 1 = a bounded wait gave up in some launch (the flag is cleared).
int conv_tc16_check_error(const tetris_filter *f) {
  Tc16State *t = static_cast<Tc16State *>(f->tc16_state);
  if (!t) return 0;
  int flag = 0;
  if (cudaMemcpy(&flag, t->d_error, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  if (flag) cudaMemset(t->d_error, 0, sizeof(int));
  return flag;
}

}  // namespace tetris
