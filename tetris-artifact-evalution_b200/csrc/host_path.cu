// The host-pointer data path: host NCHW in, host NCHW out, blocking (tetris_conv2d_host) or
// pipelined over slots (tetris_conv2d_host_async), and the workspaces both keep between calls.
#include <initializer_list>
#include <mutex>

#include "internal.h"

namespace tetris {
namespace {

constexpr int kMaxDevices = 64;

// Activation workspace of tetris_conv2d_host, one per device, grown on demand.
struct Workspace {
  std::mutex mutex;
  void *ptr = nullptr;
  size_t bytes = 0;
};
Workspace g_workspace[kMaxDevices];

// The pipelined path: `slot` selects one of kSlots (stream, workspace) pairs per device.  The copies
// of all slots go through two streams of the device, one per direction: copies of several streams
// in one direction share the link and hold back the other direction's (eight calls of 6.4 MB each
// way: 1.52 ms with the copies on the slots' own streams, 1.14 ms for the bare copies on two).
constexpr int kSlots = 4;
struct HostSlot {
  std::mutex mutex;
  cudaStream_t stream = nullptr;  // transposes and convolution
  cudaEvent_t arrived = nullptr, computed = nullptr, left = nullptr;  // input on the device; output ready; output on the host
  void *ptr = nullptr;
  size_t bytes = 0;
};
struct CopyStreams {  // made under this mutex and one slot's, destroyed under those of all slots
  std::mutex mutex;
  cudaStream_t up = nullptr, down = nullptr;
};
HostSlot g_slots[kMaxDevices][kSlots];
CopyStreams g_copy[kMaxDevices];

}  // namespace
}  // namespace tetris

using namespace tetris;

extern "C" {

int tetris_conv2d_host(const tetris_filter_t *f, const float *h_input_nchw,
                       float *h_output_nchw, int batch_size, int img_h, int img_w, int stride,
                       int padding, void *stream) {
  ConvShape s;
  int rc = make_shape(f, batch_size, img_h, img_w, stride, padding, &s);
  if (rc) return rc;
  if (batch_size == 0) return TETRIS_OK;
  if (!h_input_nchw || !h_output_nchw) { set_error("input or output pointer is NULL"); return TETRIS_ERR_INVALID; }
  DeviceGuard guard(f->device);
  if (!guard.ok) { set_error("cudaSetDevice(%d) failed", f->device); return TETRIS_ERR_CUDA; }
  cudaStream_t st = (cudaStream_t)stream;
  const size_t in_elems = (size_t)s.N * s.IC * s.H * s.W, out_elems = (size_t)s.N * s.OC * s.OH * s.OW;
  // One buffer: [input NCHW | input NHWC | output NHWC | output NCHW].  It comes from a
  // grow-only per-device workspace that is kept between calls (tetris_release_workspace frees
  // it); a call that finds the workspace in use by another thread allocates its own.
  const size_t in_pad = (in_elems + 3) / 4 * 4, out_pad = (out_elems + 3) / 4 * 4;  // (16-byte aligned parts)
  const size_t need = (2 * in_pad + 2 * out_pad) * sizeof(float);
  Workspace *ws = f->device < kMaxDevices ? &g_workspace[f->device] : nullptr;
  const bool cached = ws && ws->mutex.try_lock();
  float *d = nullptr;
  if (cached) {
    if (ws->bytes < need) {
      cudaFree(ws->ptr);
      ws->ptr = nullptr; ws->bytes = 0;
      if (cudaMalloc(&ws->ptr, need) == cudaSuccess) ws->bytes = need;
    }
    d = static_cast<float *>(ws->ptr);
  } else if (cudaMalloc(&d, need) != cudaSuccess) {
    d = nullptr;
  }
  if (!d) {
    cudaGetLastError();
    if (cached) ws->mutex.unlock();
    set_error("cudaMalloc of %zu bytes of activations failed", need);
    return TETRIS_ERR_NOMEM;
  }
  float *d_in_nchw = d, *d_in_nhwc = d + in_pad, *d_out_nhwc = d + 2 * in_pad, *d_out_nchw = d + 2 * in_pad + out_pad;
  auto done = [&](int code) {
    if (cached) ws->mutex.unlock(); else cudaFree(d);
    return code;
  };
  cudaError_t err = copy_to_device(d_in_nchw, h_input_nchw, in_elems * sizeof(float), st);
  if (err != cudaSuccess) {
    set_error("host-to-device copy failed: %s", cudaGetErrorString(err));
    return done(TETRIS_ERR_CUDA);
  }
  if ((rc = launch_nchw_to_nhwc(d_in_nchw, d_in_nhwc, s.N, s.IC, s.H, s.W, st))) return done(rc);
  if ((rc = conv_dispatch_auto(f, d_in_nhwc, d_out_nhwc, s, st))) return done(rc);
  if ((rc = launch_nhwc_to_nchw(d_out_nhwc, d_out_nchw, s.N, s.OC, s.OH, s.OW, st))) return done(rc);
  err = copy_to_host(h_output_nchw, d_out_nchw, out_elems * sizeof(float), st);
  if (err != cudaSuccess) {
    cudaGetLastError();
    set_error("convolution or device-to-host copy failed: %s", cudaGetErrorString(err));
    return done(TETRIS_ERR_CUDA);
  }
  return done(TETRIS_OK);
}

int tetris_conv2d_host_async(const tetris_filter_t *f, const float *h_input_nchw,
                             float *h_output_nchw, int batch_size, int img_h, int img_w, int stride,
                             int padding, int slot) {
  ConvShape s;
  int rc = make_shape(f, batch_size, img_h, img_w, stride, padding, &s);
  if (rc) return rc;
  if (slot < 0 || slot >= kSlots || f->device >= kMaxDevices) {
    set_error("slot %d outside [0, %d)", slot, kSlots);
    return TETRIS_ERR_INVALID;
  }
  if (batch_size == 0) return TETRIS_OK;
  if (!h_input_nchw || !h_output_nchw) { set_error("input or output pointer is NULL"); return TETRIS_ERR_INVALID; }
  DeviceGuard guard(f->device);
  if (!guard.ok) { set_error("cudaSetDevice(%d) failed", f->device); return TETRIS_ERR_CUDA; }
  HostSlot &hs = g_slots[f->device][slot];
  std::lock_guard<std::mutex> lock(hs.mutex);
  cudaStream_t up, down;  // (live while a slot's mutex is held)
  {
    CopyStreams &cs = g_copy[f->device];
    std::lock_guard<std::mutex> lock(cs.mutex);
    if (!cs.up) TETRIS_CUDA_TRY(cudaStreamCreateWithFlags(&cs.up, cudaStreamNonBlocking));
    if (!cs.down) TETRIS_CUDA_TRY(cudaStreamCreateWithFlags(&cs.down, cudaStreamNonBlocking));
    up = cs.up; down = cs.down;
  }
  if (!hs.stream) TETRIS_CUDA_TRY(cudaStreamCreateWithFlags(&hs.stream, cudaStreamNonBlocking));
  for (cudaEvent_t *e : {&hs.arrived, &hs.computed, &hs.left})
    if (!*e) TETRIS_CUDA_TRY(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
  const size_t in_elems = (size_t)s.N * s.IC * s.H * s.W, out_elems = (size_t)s.N * s.OC * s.OH * s.OW;
  const size_t in_pad = (in_elems + 3) / 4 * 4, out_pad = (out_elems + 3) / 4 * 4;
  const size_t need = (2 * in_pad + 2 * out_pad) * sizeof(float);
  if (hs.bytes < need) {
    // the slot's earlier work may still use the old buffer
    TETRIS_CUDA_TRY(cudaEventSynchronize(hs.left));
    cudaFree(hs.ptr);
    hs.ptr = nullptr; hs.bytes = 0;
    if (cudaMalloc(&hs.ptr, need) != cudaSuccess) {
      cudaGetLastError();
      set_error("cudaMalloc of %zu bytes of activations failed", need);
      return TETRIS_ERR_NOMEM;
    }
    hs.bytes = need;
  }
  float *d = static_cast<float *>(hs.ptr);
  float *d_in_nchw = d, *d_in_nhwc = d + in_pad, *d_out_nhwc = d + 2 * in_pad, *d_out_nchw = d + 2 * in_pad + out_pad;
  cudaStream_t st = hs.stream;
  // (the slot's last call has read its input buffer once `computed` has passed, its output buffer once `left` has)
  if (cudaEventQuery(hs.computed) == cudaSuccess) {
    TETRIS_CUDA_TRY(cudaMemcpyAsync(d_in_nchw, h_input_nchw, in_elems * sizeof(float), cudaMemcpyHostToDevice, up));
    TETRIS_CUDA_TRY(cudaEventRecord(hs.arrived, up));
    TETRIS_CUDA_TRY(cudaStreamWaitEvent(st, hs.arrived, 0));
  } else {  // behind the slot's own work: on the shared stream it would hold back the uploads of other slots
    TETRIS_CUDA_TRY(cudaMemcpyAsync(d_in_nchw, h_input_nchw, in_elems * sizeof(float), cudaMemcpyHostToDevice, st));
  }
  if ((rc = launch_nchw_to_nhwc(d_in_nchw, d_in_nhwc, s.N, s.IC, s.H, s.W, st))) return rc;
  if ((rc = conv_dispatch_auto(f, d_in_nhwc, d_out_nhwc, s, st))) return rc;
  TETRIS_CUDA_TRY(cudaStreamWaitEvent(st, hs.left, 0));
  if ((rc = launch_nhwc_to_nchw(d_out_nhwc, d_out_nchw, s.N, s.OC, s.OH, s.OW, st))) return rc;
  TETRIS_CUDA_TRY(cudaEventRecord(hs.computed, st));
  TETRIS_CUDA_TRY(cudaStreamWaitEvent(down, hs.computed, 0));
  TETRIS_CUDA_TRY(cudaMemcpyAsync(h_output_nchw, d_out_nchw, out_elems * sizeof(float), cudaMemcpyDeviceToHost, down));
  TETRIS_CUDA_TRY(cudaEventRecord(hs.left, down));
  return TETRIS_OK;
}

int tetris_host_sync(int device, int slot) {
  if (device < 0 || device >= kMaxDevices || slot >= kSlots) { set_error("bad device/slot"); return TETRIS_ERR_INVALID; }
  DeviceGuard guard(device);
  for (int i = 0; i < kSlots; ++i) {
    if (slot >= 0 && i != slot) continue;
    HostSlot &hs = g_slots[device][i];
    std::lock_guard<std::mutex> lock(hs.mutex);
    // the slot's stream (an aborted call may have left work there), then its last download
    if ((hs.stream && cudaStreamSynchronize(hs.stream) != cudaSuccess) || (hs.left && cudaEventSynchronize(hs.left) != cudaSuccess)) {
      set_error("pipelined convolution failed: %s", cudaGetErrorString(cudaGetLastError()));
      return TETRIS_ERR_CUDA;
    }
  }
  return TETRIS_OK;
}

void tetris_release_workspace(void) {
  int prev = -1;
  cudaGetDevice(&prev);
  for (int dev = 0; dev < kMaxDevices; ++dev) {
    Workspace &ws = g_workspace[dev];
    std::lock_guard<std::mutex> lock(ws.mutex);
    if (!ws.ptr) continue;
    if (cudaSetDevice(dev) == cudaSuccess) cudaFree(ws.ptr);
    ws.ptr = nullptr;
    ws.bytes = 0;
  }
  for (int dev = 0; dev < kMaxDevices; ++dev) {
    std::unique_lock<std::mutex> slots[kSlots];  // (a call that holds its slot's may be using the copy streams)
    for (int i = 0; i < kSlots; ++i) slots[i] = std::unique_lock<std::mutex>(g_slots[dev][i].mutex);
    for (int i = 0; i < kSlots; ++i) {
      HostSlot &hs = g_slots[dev][i];
      if (!hs.stream && !hs.ptr) continue;
      if (cudaSetDevice(dev) != cudaSuccess) continue;
      if (hs.left) cudaEventSynchronize(hs.left);
      if (hs.stream) { cudaStreamSynchronize(hs.stream); cudaStreamDestroy(hs.stream); }
      for (cudaEvent_t *e : {&hs.arrived, &hs.computed, &hs.left}) { if (*e) cudaEventDestroy(*e); *e = nullptr; }
      cudaFree(hs.ptr);
      hs.stream = nullptr; hs.ptr = nullptr; hs.bytes = 0;
    }
    CopyStreams &cs = g_copy[dev];
    std::lock_guard<std::mutex> lock(cs.mutex);
    if ((cs.up || cs.down) && cudaSetDevice(dev) == cudaSuccess) {
      if (cs.up) { cudaStreamSynchronize(cs.up); cudaStreamDestroy(cs.up); }
      if (cs.down) { cudaStreamSynchronize(cs.down); cudaStreamDestroy(cs.down); }
      cs.up = cs.down = nullptr;
    }
  }
  release_memory();
  if (prev >= 0) cudaSetDevice(prev);
}

}  // extern "C"
