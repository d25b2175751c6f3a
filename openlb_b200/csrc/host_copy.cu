// Device-to-host copies into pageable memory: staged through pinned buffers
// and written by several threads.
//
// cudaMemcpyAsync into pageable memory stages through one driver buffer and one
// thread, which also takes the page faults of memory the caller has just
// allocated (every numpy.empty).  Here the copy engine fills a ring of pinned
// buffers while threads empty it into the destination, each taking its chunk's
// faults: a chunk of 30 served cavities with their fields, 148 MB into fresh
// arrays, takes 41 ms instead of 62, 27 of them steps.  Pinned destinations and
// small copies go straight to cudaMemcpyAsync; so does a copy that finds the
// ring taken by another thread.
#include "host_copy.h"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace olb_b200 {
namespace {

constexpr size_t kChunk = size_t(512) << 10;
constexpr int kRing = 16;                        // 8 MiB of pinned memory per process
constexpr size_t kStagedFrom = size_t(1) << 20;  // below, too few chunks to overlap
constexpr int kMaxThreads = 6;

// One copy at a time (the pool's mutex).  Chunk i passes through buffer
// i % kRing: the caller issues its transfer once chunk i - kRing has left the
// buffer, a worker waits for the transfer and writes the chunk out.
class Pool {
public:
  static std::unique_ptr<Pool> make()
  {
    std::unique_ptr<Pool> p(new (std::nothrow) Pool);
    if (!p) return nullptr;
    void* base = nullptr;
    if (cudaHostAlloc(&base, kRing * kChunk, cudaHostAllocPortable) != cudaSuccess) {
      (void)cudaGetLastError();
      return nullptr;
    }
    p->base_ = static_cast<char*>(base);
    const int n = std::max(1, std::min(kMaxThreads, int(std::thread::hardware_concurrency()) - 1));
    try {  // nothing is thrown through the C interface: fewer threads, or the direct copy
      for (int k = 0; k < n; ++k) p->threads_.emplace_back([q = p.get()] { q->work(); });
    } catch (...) {
      if (p->threads_.empty()) return nullptr;
    }
    return p;
  }

  ~Pool()
  {
    {
      std::lock_guard<std::mutex> lock(mutex_);
      quit_ = true;
    }
    wake_.notify_all();
    for (std::thread& t : threads_) t.join();
    drop_events();
    if (base_) cudaFreeHost(base_);
  }

  cudaError_t copy(char* dst, const char* src, size_t bytes, int device, cudaStream_t stream)
  {
    if (device != events_device_) {  // events belong to a device
      drop_events();
      for (cudaEvent_t& ev : events_) {
        const cudaError_t e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
        if (e != cudaSuccess) {
          drop_events();
          return e;
        }
      }
      events_device_ = device;
    }
    return run(dst, src, bytes, device, stream);
  }

private:
  Pool() = default;

  void drop_events()
  {
    for (cudaEvent_t& ev : events_) {
      if (ev) cudaEventDestroy(ev);
      ev = nullptr;
    }
    events_device_ = -1;
  }

  cudaError_t run(char* dst, const char* src, size_t bytes, int device, cudaStream_t stream)
  {
    const size_t chunks = (bytes + kChunk - 1) / kChunk;
    {
      std::lock_guard<std::mutex> lock(mutex_);
      dst_ = dst;
      bytes_ = bytes;
      device_ = device;
      chunks_ = chunks;
      next_ = 0;
      issued_ = 0;
      error_ = cudaSuccess;
      for (auto& l : left_) l = 0;
      busy_ = int(threads_.size());
      ++job_;
    }
    wake_.notify_all();
    cudaError_t e = cudaSuccess;
    for (size_t i = 0; i < chunks && e == cudaSuccess; ++i) {
      const int b = int(i % kRing);
      // left_[b] counts the chunks that have left buffer b
      while (left_[b].load(std::memory_order_acquire) < i / kRing) std::this_thread::yield();
      const size_t at = i * kChunk;
      e = cudaMemcpyAsync(base_ + size_t(b) * kChunk, src + at, std::min(kChunk, bytes - at), cudaMemcpyDeviceToHost,
                          stream);
      if (e == cudaSuccess) e = cudaEventRecord(events_[b], stream);
      if (e == cudaSuccess) issued_.store(i + 1, std::memory_order_release);
    }
    if (e != cudaSuccess) stop_ = true;  // workers give up the chunks that never come
    {
      std::unique_lock<std::mutex> lock(mutex_);
      idle_.wait(lock, [&] { return busy_ == 0; });
    }
    stop_ = false;
    return e != cudaSuccess ? e : error_.load();
  }

  void work()
  {
    uint64_t seen = 0;
    for (;;) {
      {
        std::unique_lock<std::mutex> lock(mutex_);
        wake_.wait(lock, [&] { return quit_ || job_ != seen; });
        if (quit_) return;
        seen = job_;
      }
      cudaSetDevice(device_);
      for (;;) {
        const size_t i = next_.fetch_add(1);
        if (i >= chunks_) break;
        while (issued_.load(std::memory_order_acquire) <= i && !stop_) std::this_thread::yield();
        if (issued_.load(std::memory_order_acquire) <= i) break;
        const int b = int(i % kRing);
        const cudaError_t e = cudaEventSynchronize(events_[b]);
        const size_t at = i * kChunk;
        if (e == cudaSuccess) std::memcpy(dst_ + at, base_ + size_t(b) * kChunk, std::min(kChunk, bytes_ - at));
        else error_ = e;
        left_[b].fetch_add(1, std::memory_order_release);
      }
      std::lock_guard<std::mutex> lock(mutex_);
      if (--busy_ == 0) idle_.notify_all();
    }
  }

  char* base_ = nullptr;
  std::vector<std::thread> threads_;
  std::mutex mutex_;
  std::condition_variable wake_, idle_;
  bool quit_ = false;
  uint64_t job_ = 0;
  int busy_ = 0;
  // the current copy
  char* dst_ = nullptr;
  size_t bytes_ = 0, chunks_ = 0;
  int device_ = 0;
  cudaEvent_t events_[kRing] = {};
  int events_device_ = -1;
  std::atomic<size_t> next_{0}, issued_{0}, left_[kRing];
  std::atomic<cudaError_t> error_{cudaSuccess};
  std::atomic<bool> stop_{false};
};

// holders, the pool and its use; never destroyed (a handle leaked at exit
// leaves threads that wait, which the exit ends)
struct Shared {
  std::mutex mutex;         // holds, pool
  std::mutex in_use;        // one copy at a time
  int holds = 0;
  std::unique_ptr<Pool> pool;
};
Shared& shared()
{
  static Shared* s = new Shared;
  return *s;
}

} // namespace

HostCopyHold::HostCopyHold()
{
  std::lock_guard<std::mutex> lock(shared().mutex);
  ++shared().holds;
}

HostCopyHold::~HostCopyHold()
{
  std::unique_ptr<Pool> gone;
  std::lock_guard<std::mutex> lock(shared().mutex);
  if (--shared().holds == 0) gone = std::move(shared().pool);
  gone.reset();
}

cudaError_t copy_to_host(void* dst, const void* src, size_t bytes, int device, cudaStream_t stream)
{
  Shared& s = shared();
  bool staged = bytes >= kStagedFrom;
  if (staged) {
    cudaPointerAttributes attr{};
    if (cudaPointerGetAttributes(&attr, dst) != cudaSuccess) {
      (void)cudaGetLastError();
      staged = false;
    } else {
      staged = attr.type == cudaMemoryTypeUnregistered;
    }
  }
  std::unique_lock<std::mutex> use(s.in_use, std::defer_lock);
  if (staged) staged = use.try_lock();
  Pool* pool = nullptr;
  if (staged) {
    std::lock_guard<std::mutex> lock(s.mutex);
    if (!s.pool) s.pool = Pool::make();
    pool = s.pool.get();
  }
  if (!pool) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream);
  return pool->copy(static_cast<char*>(dst), static_cast<const char*>(src), bytes, device, stream);
}

} // namespace olb_b200
