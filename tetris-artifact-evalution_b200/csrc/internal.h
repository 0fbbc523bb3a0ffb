// Internal declarations of the engine: the filter handle, error plumbing and the launchers
// implemented in the individual .cu files.  Nothing here is part of the C ABI.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <vector>

#include "../../include/tetris_b200.h"
#include "format.h"

struct tetris_filter {
  int in_channel, out_channel, kernel_size, groups;
  int oc_block, tile_ic;
  int n_oc_blocks, n_stages;
  int64_t nnz, n_ops;
  int max_prog_ops;        // longest program, in records
  int device;
  uint64_t *d_ops;         // program stream (n_ops records incl. tail padding)
  int32_t *d_prog_offsets; // n_oc_blocks * n_stages + 1 record indices
  float *d_dense;          // depthwise only: dense [C][KS*KS] filter
  // LIST form (format.h), consumed by the tiled kernel
  uint64_t *d_lists;       // n_list_units 8-byte units incl. tail padding
  int32_t *d_list_offsets; // n_oc_blocks * n_stages + 1 unit indices
  int64_t n_list_units;
  int max_list_units;      // longest piece, in 8-byte units
  int deterministic;       // 1: the tensor-core variant never splits a tile's K range (no atomic adds)
  void *plan_cache;        // tiled kernel: launch plan of the last conv shape (conv_tiled.cu)
  void *tc_state;          // tensor-core variant: split dense weights + tensor maps (conv_tc.cu)
  void *tc16_state;        // split-FP16 tensor-core variant: weight images + tensor maps (conv_tc16.cu)
};

namespace tetris {

void set_error(const char *fmt, ...);

#define TETRIS_CUDA_TRY(call)                                                              \
  do {                                                                                     \
    cudaError_t err__ = (call);                                                            \
    if (err__ != cudaSuccess) {                                                            \
      ::tetris::set_error("%s failed at %s:%d: %s", #call, __FILE__, __LINE__,             \
                          cudaGetErrorString(err__));                                      \
      return TETRIS_ERR_CUDA;                                                              \
    }                                                                                      \
  } while (0)

// Overlapped launches.  A kernel that follows another on its stream may be set up -- its blocks
// placed, barriers and tensor memory made ready, weights on their way -- while the one before it
// drains: launch_overlapped marks the launch as such, grid_release in a running kernel lets the next
// one start being placed, and grid_wait returns once everything before it on the stream is complete
// and visible.  EVERY kernel launched this way calls grid_wait before it touches activations (reads
// or writes them), in at least one thread of every block on whose data all stores of that block depend:
// completion then passes on from launch to launch, and a kernel launched in the ordinary way, a
// copy or an event still sees all work before it.  What is read ahead of it is what no launch on a
// stream writes: a filter's images, complete when its creation returned.
// Activations are not read through the non-coherent path (__ldg) in these kernels: they may change
// while the kernel is resident.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// (the pointer passes through the wait, so that no load through it is moved ahead)
template <typename T> __device__ __forceinline__ T *grid_wait(T *p) {
  asm volatile("griddepcontrol.wait;" : "+l"(p) :: "memory");
  return p;
}
// Blocks of a persistent kernel call it once they hold what they need to finish (tensor memory).
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
cudaError_t launch_overlapped(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, unsigned cluster, const A &...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

struct ConvShape {
  int N, H, W, IC, OC, KS, S, P, OH, OW;
  int relu = 0;  // fused epilogue: max(y, 0) at the store (tetris_conv2d_launch_fused)
};

// Makes `device` current for the lifetime of the object and restores the previous one.
struct DeviceGuard {
  int prev = -1;
  bool ok = false;
  explicit DeviceGuard(int device) {
    if (cudaGetDevice(&prev) != cudaSuccess) return;
    ok = cudaSetDevice(device) == cudaSuccess;
  }
  ~DeviceGuard() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

// api.cu: checks the arguments of a conv call and fills in the shape
int make_shape(const tetris_filter *f, int batch, int h, int w, int stride, int padding, ConvShape *s);

// memory.cu: device memory of the filters, copies with ordinary host memory
cudaError_t device_alloc(void **p, size_t bytes);
void device_free(void *p);
cudaError_t copy_to_device(void *dst, const void *src, size_t bytes, cudaStream_t st);
cudaError_t copy_to_host(void *dst, const void *src, size_t bytes, cudaStream_t st);
void release_memory();

// compress.cu: dense filter on the device -> program stream.  The count kernel writes the length of
// every program and adds the nonzeros to *d_nnz.
int compress_count(const float *d_filter, int IC, int OC, int KS, int K, int TIC, int B, int T,
                   int32_t *d_lens, unsigned long long *d_nnz, cudaStream_t st);
// Exclusive scan of n lengths into n + 1 offsets; `meta` (may be null) receives {total, longest}.
int compress_scan(const int32_t *d_lens, int32_t *d_offsets, int n, int32_t *meta, cudaStream_t st);
int compress_fill(const float *d_filter, int IC, int OC, int KS, int K, int TIC, int B, int T,
                  const int32_t *d_offsets, uint64_t *d_ops, int64_t n_ops, cudaStream_t st);

int list_count(const float *d_filter, int IC, int OC, int KS, int K, int TIC, int B, int T,
               int32_t *d_lens, cudaStream_t st);
int list_fill(const float *d_filter, int IC, int OC, int KS, int K, int TIC, int B, int T,
              const int32_t *d_offsets, uint64_t *d_units, int64_t n_units, cudaStream_t st);

// conv_generic.cu / conv_tiled.cu / depthwise.cu / layout.cu
int launch_conv_generic(const tetris_filter *f, const float *in, float *out, const ConvShape &s,
                        cudaStream_t st);
bool conv_tiled_supported(const tetris_filter *f, const ConvShape &s);
// allow_tc: let the plan's automatic choice switch to the tensor-core variant
int launch_conv_tiled(const tetris_filter *f, const float *in, float *out, const ConvShape &s,
                      cudaStream_t st, bool allow_tc);
int tune_conv_tiled(const tetris_filter *f, const float *in, float *out, const ConvShape &s,
                    cudaStream_t st, int max_candidates, float *best_ms);
int conv_auto_choice(const tetris_filter *f, const ConvShape &s, int *variant);
void *tiled_plan_cache_new();
// The plans tetris_conv2d_tune chose, as kTunedInts ints each: the conv shape (N, H, W, S, P),
// the kernel instance, the tile shape (NSEG, TH) and whether the tensor-core variant won.
constexpr int kTunedInts = 9;
void tiled_plans_export(const tetris_filter *f, std::vector<int32_t> *out);
void tiled_plans_import(const tetris_filter *f, const int32_t *plans, int n);
// conv kernel launches issued through the library by this process (all devices, all threads)
void count_launch();
// tetris_test_inject (failure-detection tests): 1 while the tensor-core kernels are asked to leave
// out every CTA's first activation load, with the poll limit their barrier waits then use.
int test_injection(unsigned *spin_limit);
void tiled_plan_cache_delete(void *cache);
// weights.cu: the tensor-core kernels' weight images of a filter, where they cover it
struct WeightImages {
  float *tc = nullptr;            // split TF32
  int bn = 128;                   // ... channels of its tiles
  void *tc16 = nullptr;           // split FP16
  int stack = 0;                  // ... w_hi and w_lo stacked (at most 64 output channels)
  const float *scale = nullptr;   // ... per output channel
};
int tensor_prepare(tetris_filter *f, const float *d_dense);
// the variants' shares of it: buffers, scales, folded stems; what is left to build goes into `w`
int conv_tc_prepare(tetris_filter *f, const float *d_dense, WeightImages *w);
void conv_tc_state_delete(void *state);
bool conv_tc_supported(const tetris_filter *f, const ConvShape &s);
int launch_conv_tc(const tetris_filter *f, const float *in, float *out, const ConvShape &s,
                   cudaStream_t st);
int conv_tc_check_error(const tetris_filter *f);
int conv_tc16_prepare(tetris_filter *f, const float *d_dense, WeightImages *w);
void conv_tc16_state_delete(void *state);
bool conv_tc16_supported(const tetris_filter *f, const ConvShape &s);
double conv_tc16_cost(const tetris_filter *f, const ConvShape &s);  // estimated clocks of a launch, negative: not covered
int launch_conv_tc16(const tetris_filter *f, const float *in, float *out, const ConvShape &s, cudaStream_t st);
int conv_tc16_check_error(const tetris_filter *f);
int launch_depthwise(const tetris_filter *f, const float *in, float *out, const ConvShape &s,
                     cudaStream_t st);
int depthwise_check_error();
// chain.cu / api.cu: y = max(y, 0) in place; an automatic launch of one conv (with its fused
// options in s); whether the launch at hand rectified at its own store
int launch_relu_inplace(float *y, size_t n, cudaStream_t st);
int conv_dispatch_auto(const tetris_filter *f, const float *in, float *out, const ConvShape &s, cudaStream_t st);
void note_relu_fused();
int launch_nchw_to_nhwc(const float *src, float *dst, int N, int C, int H, int W, cudaStream_t st);
int launch_nhwc_to_nchw(const float *src, float *dst, int N, int C, int H, int W, cudaStream_t st);

}  // namespace tetris
