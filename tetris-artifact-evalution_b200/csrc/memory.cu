// Device memory of the filters and copies between the device and ordinary host memory.
//
// Filters take their device memory from one stream-ordered pool per device: a cudaMalloc costs
// 10-100 us and a cudaFree waits for the device, and a filter has a dozen buffers (512 x 512 x 3 x 3:
// 5 ms to create, most of it in the allocator).  Up to 256 MB of freed memory stay with the pool;
// tetris_release_workspace gives them back.
//
// Ordinary (pageable) host memory.  A copy between it and the device runs through the driver's own
// bounce buffer on the calling thread, at the speed of one core's memcpy (15 GB/s on a host whose
// link carries 55): 210 us for 3.2 MB each way, against 58 us of DMA.  Here a few threads move chunks
// between the caller's array and a page-locked ring while the copy engine moves the chunks before
// them, so that the link sets the pace.  Page-locked arrays are copied from and to directly.
#include <string.h>
#if defined(__x86_64__)
#include <emmintrin.h>
#endif

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

#include "internal.h"

namespace tetris {
namespace {

constexpr int kMaxDevices = 64;
constexpr uint64_t kKeptBytes = (uint64_t)256 << 20;

struct DevicePool {
  std::mutex mutex;
  cudaMemPool_t pool = nullptr;
};
DevicePool g_pools[kMaxDevices];

// ---- chunked copies through page-locked memory -------------------------------------------------
constexpr int kRing = 32;                          // chunks in flight per direction
constexpr size_t kMaxChunk = (size_t)512 << 10, kMinChunk = (size_t)64 << 10;
// Smaller copies are left to the driver: waking the helpers for an upload of 288 to 640 KB cost a blocking call 10 to
// 16 us more than the driver's copy of it (512 KB each way 129 us, 112 with the upload left to the driver, 117 with
// both); from 768 KB on the ring is ahead (91 us against 100), and for downloads from 256 KB on.
constexpr size_t kStagedUpload = (size_t)768 << 10, kStagedDownload = (size_t)256 << 10;

inline void relax() {
#if defined(__x86_64__)
  __builtin_ia32_pause();
#endif
}

// memcpy into page-locked memory that a copy engine reads next (dst 16-byte aligned).  The stores go past the caches: the
// copy engine reads lines that lie modified in other cores' caches slowly once those cores sleep (a blocking call
// with 4 MB in and 64 KB out, whose helpers sleep while it computes: 670 us, 178 with these stores, 290 by the
// driver; 4 MB each way, where they do not, 370, 317 and 500).
inline void copy_past_caches(char *dst, const char *src, size_t n) {
#if defined(__x86_64__)
  size_t i = 0;
  for (; i + 64 <= n; i += 64) {
    const __m128i a = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + i)), b = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + i + 16));
    const __m128i c = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + i + 32)), d = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + i + 48));
    _mm_stream_si128(reinterpret_cast<__m128i *>(dst + i), a);
    _mm_stream_si128(reinterpret_cast<__m128i *>(dst + i + 16), b);
    _mm_stream_si128(reinterpret_cast<__m128i *>(dst + i + 32), c);
    _mm_stream_si128(reinterpret_cast<__m128i *>(dst + i + 48), d);
  }
  memcpy(dst + i, src + i, n - i);
  _mm_sfence();  // (before the flag that says the chunk is there)
#else
  memcpy(dst, src, n);
#endif
}

struct Job {
  char *user;                     // the caller's array
  char *ring;                     // page-locked chunks
  size_t bytes, chunk;
  int n;                          // chunks
  bool to_ring;
  std::atomic<int> next{0};       // first chunk nobody has taken
  std::atomic<int> ready{0};      // chunks below this may be taken
  // chunk i has been moved: flag i % kRing, taken back by the caller before chunk i + kRing is ready
  std::atomic<unsigned char> done[kRing] = {};
  std::atomic<int> users{0};      // threads that hold a pointer to this job

  bool available() const { return next.load() < n && next.load() < ready.load(); }
  // Takes and moves one chunk; false if none may be taken now.
  bool work() {
    int i = next.load(std::memory_order_relaxed);
    do {
      if (i >= n || i >= ready.load(std::memory_order_acquire)) return false;
    } while (!next.compare_exchange_weak(i, i + 1, std::memory_order_relaxed));
    char *u = user + (size_t)i * chunk, *r = ring + (size_t)(i % kRing) * kMaxChunk;
    const size_t len = std::min(chunk, bytes - (size_t)i * chunk);
    if (to_ring) copy_past_caches(r, u, len); else memcpy(u, r, len);
    done[i % kRing].store(1, std::memory_order_release);
    return true;
  }
  bool take_done(int i) {
    if (!done[i % kRing].load(std::memory_order_acquire)) return false;
    done[i % kRing].store(0, std::memory_order_relaxed);
    return true;
  }
};

// One per device, made at the first staged copy and never destroyed (its threads may outlive static
// destructors); release() gives the threads and the memory back.
class Stager {
 public:
  std::mutex in_use;              // one staged copy at a time; others go through the driver

  bool open() {
    if (ring_in_) return true;
    if (cudaHostAlloc((void **)&ring_in_, 2 * kRing * kMaxChunk, cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      ring_in_ = nullptr;
      return false;
    }
    ring_out_ = ring_in_ + kRing * kMaxChunk;
    for (int i = 0; i < kRing; ++i)
      if (cudaEventCreateWithFlags(&events_[i], cudaEventDisableTiming) != cudaSuccess) {
        cudaGetLastError();
        release();
        return false;
      }
    if (cudaEventCreateWithFlags(&uploaded_, cudaEventDisableTiming) != cudaSuccess) { cudaGetLastError(); release(); return false; }
    // four cores move as much as the link carries; the caller is one more.  All devices together take a third
    // of the host's cores; on a device that comes too late for them the caller moves the chunks alone.
    const int most = std::max(1, (int)(std::thread::hardware_concurrency() / 3));
    stop_ = false;
    try {
      while (threads_.size() < 4) {
        if (helpers_.fetch_add(1) >= most) { helpers_.fetch_sub(1); break; }
        try {
          threads_.emplace_back([this] { serve(); });
        } catch (...) {
          helpers_.fetch_sub(1);
          throw;
        }
      }
    } catch (...) {
    }
    return true;
  }

  void release() {
    { std::lock_guard<std::mutex> lock(mutex_); stop_ = true; }
    wake_.notify_all();
    for (std::thread &t : threads_) t.join();
    helpers_.fetch_sub((int)threads_.size());
    threads_.clear();
    if (uploaded_) { cudaEventSynchronize(uploaded_); cudaEventDestroy(uploaded_); uploaded_ = nullptr; }
    for (cudaEvent_t &e : events_) { if (e) cudaEventDestroy(e); e = nullptr; }
    cudaFreeHost(ring_in_);
    ring_in_ = ring_out_ = nullptr;
  }

  // Whether an upload on `st` may use the ring now: the last upload has left it, or is on `st` as well, where this one
  // comes behind it whichever way it goes.  (On another stream it may stand behind any amount of work.)
  bool ring_free(cudaStream_t st) { return st == last_ || cudaEventQuery(uploaded_) != cudaErrorNotReady; }

  // The caller's array -> device; when this returns the array may be reused, the last copies out of
  // the ring may still be under way on `st`.
  cudaError_t upload(void *dst, const void *src, size_t bytes, cudaStream_t st) {
    cudaError_t err = cudaEventSynchronize(uploaded_);  // (the last upload has left the ring)
    if (err != cudaSuccess) return err;
    Job job;
    prepare(&job, static_cast<char *>(const_cast<void *>(src)), ring_in_, bytes, true);
    job.ready.store(std::min(job.n, kRing));
    post(&job);
    for (int sent = 0, back = 0; sent < job.n && err == cudaSuccess;) {
      if (job.take_done(sent)) {
        const size_t at = (size_t)sent * job.chunk;
        err = cudaMemcpyAsync(static_cast<char *>(dst) + at, job.ring + (size_t)(sent % kRing) * kMaxChunk,
                              std::min(job.chunk, bytes - at), cudaMemcpyHostToDevice, st);
        if (err == cudaSuccess && job.n > kRing) err = cudaEventRecord(events_[sent % kRing], st);
        ++sent;
      } else if (back < sent && back + kRing < job.n) {
        const cudaError_t q = cudaEventQuery(events_[back % kRing]);
        if (q == cudaSuccess) make_ready(&job, std::min(job.n, ++back + kRing));  // that chunk of the ring is free again
        else if (q != cudaErrorNotReady) err = q;
        else if (!job.work()) relax();
      } else if (!job.work()) {
        relax();
      }
    }
    finish(&job);
    const cudaError_t marked = cudaEventRecord(uploaded_, st);
    last_ = st;
    if (err == cudaSuccess) return marked;
    cudaStreamSynchronize(st);  // (copies out of the ring may be under way)
    return err;
  }

  // Device -> the caller's array, behind what `st` holds; complete when this returns.
  cudaError_t download(void *dst, const void *src, size_t bytes, cudaStream_t st) {
    Job job;
    prepare(&job, static_cast<char *>(dst), ring_out_, bytes, false);
    cudaError_t err = cudaSuccess;
    int sent = 0, landed = 0;
    auto send = [&]() {
      const size_t at = (size_t)sent * job.chunk;
      err = cudaMemcpyAsync(job.ring + (size_t)(sent % kRing) * kMaxChunk, static_cast<const char *>(src) + at,
                            std::min(job.chunk, bytes - at), cudaMemcpyDeviceToHost, st);
      if (err == cudaSuccess) err = cudaEventRecord(events_[sent % kRing], st);
      ++sent;
    };
    while (sent < std::min(job.n, kRing) && err == cudaSuccess) send();
    post(&job);
    for (int moved = 0; moved < job.n && err == cudaSuccess;) {
      if (job.take_done(moved)) {
        if (sent < job.n && sent - moved <= kRing) send();  // (chunk `moved` of the ring is free again)
        ++moved;
      } else if (landed < sent) {
        const cudaError_t q = cudaEventQuery(events_[landed % kRing]);
        if (q == cudaSuccess) make_ready(&job, ++landed);
        else if (q != cudaErrorNotReady) err = q;
        else if (!job.work()) relax();
      } else if (!job.work()) {
        relax();
      }
    }
    finish(&job);
    if (err != cudaSuccess) cudaStreamSynchronize(st);  // (copies into the ring may be under way)
    return err;
  }

 private:
  void prepare(Job *job, char *user, char *ring, size_t bytes, bool to_ring) {
    job->user = user; job->ring = ring; job->bytes = bytes; job->to_ring = to_ring;
    // eight chunks or more, so that the first copy starts early and the last one is short
    job->chunk = std::min(kMaxChunk, std::max(kMinChunk, (bytes / 8 + 4095) / 4096 * 4096));
    job->n = (int)((bytes + job->chunk - 1) / job->chunk);
  }
  void post(Job *job) {
    { std::lock_guard<std::mutex> lock(mutex_); job_ = job; ++jobs_; }
    wake_.notify_all();
  }
  void make_ready(Job *job, int chunks) {
    job->ready.store(chunks);
    if (sleepers_.load() == 0) return;
    { std::lock_guard<std::mutex> lock(mutex_); }  // (a helper that has just found nothing to do is waiting by now)
    wake_.notify_one();
  }
  void finish(Job *job) {  // nobody takes another chunk, and nobody is left inside the job
    job->next.store(job->n, std::memory_order_relaxed);
    { std::lock_guard<std::mutex> lock(mutex_); job_ = nullptr; }
    while (job->users.load(std::memory_order_acquire)) relax();
  }
  // A helper joins each copy once and looks for chunks for about 250 us; when the device has not got that far
  // it sleeps until there is one.
  void serve() {
    std::unique_lock<std::mutex> lock(mutex_);
    for (unsigned joined = 0;;) {
      sleepers_.fetch_add(1);
      wake_.wait(lock, [&] { return stop_ || (job_ && (jobs_ != joined || job_->available())); });
      sleepers_.fetch_sub(1);
      if (stop_) return;
      Job *job = job_;
      joined = jobs_;
      job->users.fetch_add(1, std::memory_order_relaxed);
      lock.unlock();
      for (int idle = 0; idle < 5000 && job->next.load(std::memory_order_relaxed) < job->n;) {
        if (job->work()) idle = 0;
        else { ++idle; relax(); }
      }
      job->users.fetch_sub(1, std::memory_order_release);
      lock.lock();
    }
  }

  std::mutex mutex_;
  std::condition_variable wake_;
  Job *job_ = nullptr;
  unsigned jobs_ = 0;             // copies so far
  std::atomic<int> sleepers_{0};
  static std::atomic<int> helpers_;  // of all devices
  bool stop_ = false;
  std::vector<std::thread> threads_;
  char *ring_in_ = nullptr, *ring_out_ = nullptr;
  cudaEvent_t events_[kRing] = {}, uploaded_ = nullptr;
  cudaStream_t last_ = nullptr;   // of the last upload
};

std::atomic<int> Stager::helpers_{0};

std::mutex g_stagers_mutex;
Stager *g_stagers[kMaxDevices];

Stager *stager_of(int device) {
  if (device >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lock(g_stagers_mutex);
  if (!g_stagers[device]) g_stagers[device] = new (std::nothrow) Stager();
  return g_stagers[device];
}

bool pageable(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return true; }
  return a.type == cudaMemoryTypeUnregistered;
}

// Whether a copy of `bytes` with this host array goes through the ring; the stager then is in use.
Stager *take_stager(const void *host, size_t bytes, size_t at_least) {
  int dev = 0;
  if (bytes < at_least || !pageable(host) || cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  Stager *s = stager_of(dev);
  if (!s || !s->in_use.try_lock()) return nullptr;
  if (s->open()) return s;
  s->in_use.unlock();
  return nullptr;
}

}  // namespace

// `bytes` from the pool of the current device, ready on every stream.
cudaError_t device_alloc(void **p, size_t bytes) {
  *p = nullptr;
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  if (dev >= kMaxDevices) return cudaMalloc(p, bytes);
  DevicePool &dp = g_pools[dev];
  {
    std::lock_guard<std::mutex> lock(dp.mutex);
    if (!dp.pool) {
      cudaMemPoolProps props = {};
      props.allocType = cudaMemAllocationTypePinned;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = dev;
      if ((err = cudaMemPoolCreate(&dp.pool, &props)) != cudaSuccess) { dp.pool = nullptr; return err; }
      uint64_t keep = kKeptBytes;
      cudaMemPoolSetAttribute(dp.pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
  }
  // (allocated, used and freed in the order of the default stream; other streams see a filter only
  // once its creation has been waited for)
  return cudaMallocFromPoolAsync(p, std::max<size_t>(bytes, 1), dp.pool, 0);
}

// Nothing on the device may still use `p` (tetris_filter_destroy waits for the device).
void device_free(void *p) {
  if (p) cudaFreeAsync(p, 0);
}

// Host -> device in the order of `st`; `src` may be reused when this returns (unless it is
// page-locked: then once `st` has passed).
cudaError_t copy_to_device(void *dst, const void *src, size_t bytes, cudaStream_t st) {
  Stager *s = take_stager(src, bytes, kStagedUpload);
  if (s && !s->ring_free(st)) {
    s->in_use.unlock();
    s = nullptr;
  }
  if (!s) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
  const cudaError_t err = s->upload(dst, src, bytes, st);
  s->in_use.unlock();
  return err;
}

// Device -> host behind what `st` holds; complete when this returns.
cudaError_t copy_to_host(void *dst, const void *src, size_t bytes, cudaStream_t st) {
  Stager *s = take_stager(dst, bytes, kStagedDownload);
  if (s) {
    const cudaError_t err = s->download(dst, src, bytes, st);
    s->in_use.unlock();
    return err;
  }
  const cudaError_t err = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
  return err == cudaSuccess ? cudaStreamSynchronize(st) : err;
}

// Gives back the rings, their threads and what the pools keep.
void release_memory() {
  int prev = -1;
  cudaGetDevice(&prev);
  {
    std::lock_guard<std::mutex> lock(g_stagers_mutex);
    for (int dev = 0; dev < kMaxDevices; ++dev) {
      if (!g_stagers[dev]) continue;
      std::lock_guard<std::mutex> use(g_stagers[dev]->in_use);
      if (cudaSetDevice(dev) == cudaSuccess) g_stagers[dev]->release();
    }
  }
  for (int dev = 0; dev < kMaxDevices; ++dev) {
    std::lock_guard<std::mutex> lock(g_pools[dev].mutex);
    if (g_pools[dev].pool && cudaSetDevice(dev) == cudaSuccess) {
      cudaDeviceSynchronize();
      cudaMemPoolTrimTo(g_pools[dev].pool, 0);
    }
  }
  if (prev >= 0) cudaSetDevice(prev);
}

}  // namespace tetris
