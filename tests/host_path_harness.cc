// Runs host_path.cu and memory.cu on the CPU: the CUDA runtime calls they make are answered here, by a
// model of streams and events that says when a handle is used after its end and lets a scenario decide what
// an event's query returns.  Built with the two files by tests/test_host_path_cpu.py; the first argument names
// the scenario, exit code 0 means that it went as it should.
#include <cuda_runtime.h>
#include <stdio.h>
#include <string.h>
#include <time.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <functional>
#include <mutex>
#include <new>
#include <set>
#include <string>
#include <thread>
#include <vector>

#include "../tetris-artifact-evalution_b200/csrc/internal.h"

// ---- the model ----------------------------------------------------------------------------------
static std::mutex g_model;
static std::set<void *> g_streams, g_events, g_recorded;
static cudaStream_t g_last_upload = nullptr;
static std::atomic<size_t> g_handles{0x1000};
static std::atomic<int> g_faults{0}, g_queries{0}, g_waits{0}, g_ring_copies{0}, g_direct_copies{0};
static std::function<cudaError_t(cudaEvent_t)> g_query;          // answers cudaEventQuery
static std::function<cudaError_t(cudaEvent_t)> g_event_sync;     // answers cudaEventSynchronize
static std::function<void(cudaStream_t)> g_on_wait, g_on_sync;   // called before these are answered
static const char *g_ring = nullptr;
static size_t g_ring_bytes = 0;

static std::atomic<bool> g_no_memory{false};  // operator new fails
void *operator new(size_t n) {
  void *p = g_no_memory ? nullptr : malloc(n ? n : 1);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }

static void use_stream(cudaStream_t s) {
  std::lock_guard<std::mutex> lock(g_model);
  if (s && !g_streams.count(s)) { fprintf(stderr, "a stream was used after its end\n"); ++g_faults; }
}
static void use_event(cudaEvent_t e) {
  std::lock_guard<std::mutex> lock(g_model);
  if (!g_events.count(e)) { fprintf(stderr, "an event was used after its end\n"); ++g_faults; }
}
static bool in_ring(const void *p) { return g_ring && (const char *)p >= g_ring && (const char *)p < g_ring + g_ring_bytes; }

extern "C" {
static thread_local int t_device = 0;
cudaError_t cudaGetDevice(int *d) { *d = t_device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { t_device = d; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = (cudaStream_t)(g_handles += 16);
  std::lock_guard<std::mutex> lock(g_model);
  g_streams.insert(*s);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  use_stream(s);
  std::lock_guard<std::mutex> lock(g_model);
  g_streams.erase(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { use_stream(s); if (g_on_sync) g_on_sync(s); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  if (g_on_wait) g_on_wait(s);
  ++g_waits;
  use_stream(s); use_event(e);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  *e = (cudaEvent_t)(g_handles += 16);
  std::lock_guard<std::mutex> lock(g_model);
  g_events.insert(*e);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  use_event(e);
  std::lock_guard<std::mutex> lock(g_model);
  g_events.erase(e); g_recorded.erase(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  use_event(e); use_stream(s);
  std::lock_guard<std::mutex> lock(g_model);
  g_recorded.insert(e);
  return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
  use_event(e);
  ++g_queries;
  std::unique_lock<std::mutex> lock(g_model);
  if (!g_recorded.count(e)) return cudaSuccess;
  lock.unlock();
  return g_query ? g_query(e) : cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) { use_event(e); return g_event_sync ? g_event_sync(e) : cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind kind, cudaStream_t st) {
  use_stream(st);
  if (kind == cudaMemcpyHostToDevice) g_last_upload = st;
  ++(in_ring(d) || in_ring(s) ? g_ring_copies : g_direct_copies);
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) { *p = malloc(n); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
  *p = malloc(n);
  g_ring = (const char *)*p; g_ring_bytes = n;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { free(p); g_ring = nullptr; return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) { a->type = cudaMemoryTypeUnregistered; return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) { *p = (cudaMemPool_t)16; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
}

// ---- what the two files take from the rest of the library: a 1x1 layer that copies its input ------
namespace tetris {
static thread_local std::string g_message;
void set_error(const char *fmt, ...) { g_message = fmt; }
int make_shape(const tetris_filter *f, int n, int h, int w, int stride, int pad, ConvShape *s) {
  s->N = n; s->H = s->OH = h; s->W = s->OW = w; s->IC = f->in_channel; s->OC = f->out_channel; s->KS = 1; s->S = stride; s->P = pad;
  return TETRIS_OK;
}
static int copy(const float *a, float *b, size_t n) { memcpy(b, a, n * sizeof(float)); return TETRIS_OK; }
int launch_nchw_to_nhwc(const float *a, float *b, int N, int C, int H, int W, cudaStream_t st) { use_stream(st); return copy(a, b, (size_t)N * C * H * W); }
int launch_nhwc_to_nchw(const float *a, float *b, int N, int C, int H, int W, cudaStream_t st) { use_stream(st); return copy(a, b, (size_t)N * C * H * W); }
int conv_dispatch_auto(const tetris_filter *, const float *a, float *b, const ConvShape &s, cudaStream_t st) {
  use_stream(st);
  return copy(a, b, (size_t)s.N * s.OC * s.OH * s.OW);
}
}  // namespace tetris

using namespace std::chrono_literals;
struct Signal {  // set once; waited for with a limit
  std::mutex m;
  std::condition_variable cv;
  bool on = false;
  void set() { { std::lock_guard<std::mutex> l(m); on = true; } cv.notify_all(); }
  void wait(std::chrono::milliseconds limit) { std::unique_lock<std::mutex> l(m); cv.wait_for(l, limit, [this] { return on; }); }
};

static tetris_filter make_filter(int c) {
  tetris_filter f = {};
  f.in_channel = f.out_channel = c; f.kernel_size = f.groups = 1;
  return f;
}
static std::vector<float> ramp(size_t n) {
  std::vector<float> v(n);
  for (size_t i = 0; i < n; ++i) v[i] = (float)(i % 977);
  return v;
}

// tetris_release_workspace on one thread, behind the first slots, while a call on another thread begins
static int release_race() {
  tetris_filter f = make_filter(4);
  const auto x = ramp(4 * 9);
  std::vector<float> y(x.size());
  if (tetris_conv2d_host_async(&f, x.data(), y.data(), 1, 3, 3, 1, 0, 3)) return 1;
  Signal at_last_slot, in_call, released;
  const std::thread::id self = std::this_thread::get_id();
  g_on_sync = [&](cudaStream_t) {
    if (std::this_thread::get_id() != self) { at_last_slot.set(); in_call.wait(500ms); }
  };
  g_on_wait = [&](cudaStream_t) {
    if (std::this_thread::get_id() == self) { in_call.set(); released.wait(500ms); }
  };
  std::thread other([&] { tetris_release_workspace(); released.set(); });
  at_last_slot.wait(2000ms);
  const int rc = tetris_conv2d_host_async(&f, x.data(), y.data(), 1, 3, 3, 1, 0, 0);
  other.join();
  g_on_sync = g_on_wait = nullptr;
  return rc || g_faults ? 1 : 0;
}

// An event reports an error of the device: the call returns it, whichever way the data goes, and the next
// call is served.  The first array is larger than the ring, the chunks that went round it are watched by events.
static int device_error(bool upload) {
  tetris_filter f = make_filter(16);
  const int h = 700;
  const auto x = ramp((size_t)16 * h * h);
  std::vector<float> y(x.size(), -1.f);
  if (tetris_conv2d_host(&f, x.data(), y.data(), 1, h, h, 1, 0, nullptr) || y != x || g_ring_copies == 0) return 1;
  const int before = g_queries;
  const int fail_at = upload ? 5 : 40;
  g_query = [&](cudaEvent_t) { return g_queries - before >= fail_at ? cudaErrorIllegalAddress : cudaSuccess; };
  if (tetris_conv2d_host(&f, x.data(), y.data(), 1, h, h, 1, 0, nullptr) != TETRIS_ERR_CUDA) return 1;
  g_query = nullptr;
  y.assign(y.size(), -1.f);
  return tetris_conv2d_host(&f, x.data(), y.data(), 1, h, h, 1, 0, nullptr) || y != x || g_faults;
}

// The upload before this one ended in an error: so does this call
static int upload_mark_error() {
  tetris_filter f = make_filter(16);
  const auto x = ramp((size_t)16 * 128 * 128);
  std::vector<float> y(x.size());
  if (tetris_conv2d_host(&f, x.data(), y.data(), 1, 128, 128, 1, 0, nullptr) || y != x) return 1;
  g_event_sync = [](cudaEvent_t) { return cudaErrorIllegalAddress; };
  return tetris_conv2d_host(&f, x.data(), y.data(), 1, 128, 128, 1, 0, nullptr) != TETRIS_ERR_CUDA;
}

// A staged copy, once the ring is there, takes no memory: nothing to throw through the C entry
static int no_memory() {
  tetris_filter f = make_filter(16);
  const int h = 700;
  const auto x = ramp((size_t)16 * h * h);
  std::vector<float> y(x.size());
  if (tetris_conv2d_host(&f, x.data(), y.data(), 1, h, h, 1, 0, nullptr) || y != x) return 1;
  y.assign(y.size(), -1.f);
  g_no_memory = true;
  const int rc = tetris_conv2d_host(&f, x.data(), y.data(), 1, h, h, 1, 0, nullptr);
  g_no_memory = false;
  return rc || y != x;
}

// While the device computes, the helpers of a download sleep: the call takes the processor time of its own thread
static int idle_helpers() {
  tetris_filter f = make_filter(16);
  const int h = 200;
  const auto x = ramp((size_t)16 * h * h);
  std::vector<float> y(x.size());
  if (tetris_conv2d_host(&f, x.data(), y.data(), 1, h, h, 1, 0, nullptr) || y != x) return 1;
  const auto busy_until = std::chrono::steady_clock::now() + 400ms;
  g_query = [&](cudaEvent_t) { return std::chrono::steady_clock::now() < busy_until ? cudaErrorNotReady : cudaSuccess; };
  y.assign(y.size(), -1.f);
  const clock_t before = clock();
  if (tetris_conv2d_host(&f, x.data(), y.data(), 1, h, h, 1, 0, nullptr) || y != x) return 1;
  const double used = (double)(clock() - before) / CLOCKS_PER_SEC;
  fprintf(stderr, "%.2f s of processor time\n", used);
  return used > 0.6;
}

static int threads_of_process() {
  FILE *fh = fopen("/proc/self/status", "r");
  char line[256];
  int n = -1;
  while (fh && fgets(line, sizeof(line), fh)) sscanf(line, "Threads: %d", &n);
  if (fh) fclose(fh);
  return n;
}

// The helpers of all devices together are at most a third of the cores, and a release gives them back
static int helper_budget() {
  const auto x = ramp((size_t)16 * 200 * 200);
  std::vector<float> y(x.size());
  const int most = std::max(1, (int)std::thread::hardware_concurrency() / 3);
  for (int round = 0; round < 2; ++round) {
    for (int dev = 0; dev < 8; ++dev) {
      tetris_filter f = make_filter(16);
      f.device = dev;
      y.assign(y.size(), -1.f);
      if (tetris_conv2d_host(&f, x.data(), y.data(), 1, 200, 200, 1, 0, nullptr) || y != x) return 1;
    }
    const int n = threads_of_process();
    fprintf(stderr, "%d threads, %d cores\n", n, (int)std::thread::hardware_concurrency());
    if (n < 2 || n > 1 + most) return 1;
    tetris_release_workspace();
    if (threads_of_process() != 1) return 1;
  }
  return 0;
}

// The last upload is still on its way on one stream: an upload on another stream does not wait for it
static int busy_ring() {
  tetris_filter f = make_filter(64);
  f.out_channel = 1;
  const auto x = ramp((size_t)64 * 64 * 64);
  std::vector<float> y(64 * 64);
  cudaStream_t a, b;
  cudaStreamCreateWithFlags(&a, 0);
  cudaStreamCreateWithFlags(&b, 0);
  auto call = [&](cudaStream_t s) { return tetris_conv2d_host(&f, x.data(), y.data(), 1, 64, 64, 1, 0, s); };
  if (call(a) || g_ring_copies == 0) return 1;
  int waits = 0;
  g_query = [](cudaEvent_t) { return cudaErrorNotReady; };
  g_event_sync = [&](cudaEvent_t) { ++waits; return cudaSuccess; };
  const int staged = g_ring_copies;
  if (call(b) || g_ring_copies != staged || waits) return 1;  // by the driver, at once
  if (call(a) || g_ring_copies == staged || !waits) return 1;  // behind its own upload
  return g_faults;
}

// A slot that is used again while it works does not hold back the upload of an idle one
static int slot_in_use() {
  tetris_filter f = make_filter(4);
  const auto x = ramp(4 * 9);
  std::vector<float> y(x.size());
  auto call = [&](int slot) { return tetris_conv2d_host_async(&f, x.data(), y.data(), 1, 3, 3, 1, 0, slot); };
  if (call(0)) return 1;
  const cudaStream_t shared = g_last_upload;
  g_query = [](cudaEvent_t) { return cudaErrorNotReady; };
  int waits = 0;
  g_on_wait = [&](cudaStream_t s) { waits += s == shared; };
  if (call(0) || g_last_upload == shared) return 1;  // on its own stream
  if (call(1) || g_last_upload != shared) return 1;  // idle: on the shared one, which waits for nobody
  g_query = nullptr;
  if (call(0) || g_last_upload != shared) return 1;
  return waits || g_faults;
}

int main(int argc, char **argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  if (what == "release_race") return release_race();
  if (what == "upload_error") return device_error(true);
  if (what == "download_error") return device_error(false);
  if (what == "upload_mark_error") return upload_mark_error();
  if (what == "no_memory") return no_memory();
  if (what == "idle_helpers") return idle_helpers();
  if (what == "helper_budget") return helper_budget();
  if (what == "busy_ring") return busy_ring();
  if (what == "slot_in_use") return slot_in_use();
  fprintf(stderr, "unknown scenario\n");
  return 2;
}
