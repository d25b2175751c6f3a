// Device-to-host copies into pageable memory: staged through pinned buffers
// and written by several threads.
//
// cudaMemcpyAsync into pageable memory stages through one driver buffer and one
// thread, which also takes the page faults of memory the caller has just
// allocated (every numpy.empty).  Here the copy engine fills a ring of pinned
// buffers while threads empty it into the destination, each taking its chunk's
// faults.  268 MB of 256^3 density and velocity on a 16-core host: 16 ms into
// fresh arrays (57 direct), 8 into arrays used before (16 direct); with two
// cores 38 (57) and 18 (16).  The fields of 30 served cavities, 148 MB in 60
// copies: 23 ms fresh (64 direct), 8.3 reused (10.5).  Pinned destinations and
// small copies go straight to cudaMemcpyAsync; so does a copy that finds the
// ring taken by another thread.
//
// One thread waits for the device: the caller, as with a direct copy.  The copy
// threads sleep until the first chunk is there, so a copy called behind a long
// solve keeps one core waiting, not all of theirs.
#include "host_copy.h"

#include <pthread.h>
#include <sched.h>
#include <sys/mman.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace olb_b200 {
namespace {

constexpr size_t kChunk = size_t(512) << 10;
constexpr size_t kRing = 16;                     // 8 MiB of pinned memory per process
constexpr size_t kStagedFrom = size_t(1) << 20;  // below, too few chunks to overlap
constexpr size_t kHugePage = size_t(2) << 20;
constexpr size_t kMapped = kRing * kChunk + kHugePage;
// Making the ring and its threads and giving them back takes 1.5 ms (7 to 12 with
// cudaHostAlloc, which pins 4 KiB pages), as much as staging saves on 10 MB of
// fresh or 50 MB of reused memory.  They are made by the copy that brings what the
// handles now alive have copied to this, so a program with a handle per small
// solve pays nothing (96^3 lattice made, 10 steps, fields fetched, closed: 6 ms,
// 15 with a ring every time).
constexpr size_t kRingFrom = size_t(32) << 20;
constexpr int kMaxThreads = 6;
// how long a thread looks for the next chunk (or the caller for a free buffer)
// before it sleeps: chunks land every 10 us, waking takes several times that, and
// the copies of a served chunk follow one another in 100 us (six cavities of 20..60
// with their fields 2.01 ms with 50 us, 1.71 with 300; thirty of 24..96 50.9 and 49.0)
constexpr std::chrono::microseconds kLook{300};

// One copy at a time (Shared::in_use).  Chunk i passes through buffer i % kRing:
// the caller issues its transfer once chunk i - kRing has left the buffer,
// waits for the transfers in order and hands out each chunk as it lands; any
// thread, the caller too when it has nothing to issue or wait for, writes it out.
class Pool {
public:
  static std::unique_ptr<Pool> make()
  {
    std::unique_ptr<Pool> p(new (std::nothrow) Pool);
    if (!p) return nullptr;
    // mapped apart, so that the caller's heap stays as it is
    void* const map = mmap(nullptr, kMapped, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (map == MAP_FAILED) return nullptr;
    p->map_ = map;
    p->base_ = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(map) + kHugePage - 1) / kHugePage * kHugePage);
    (void)madvise(p->base_, kRing * kChunk, MADV_HUGEPAGE);  // four pages to pin, not 2048
    std::memset(p->base_, 0, kRing * kChunk);
    p->pinned_ = cudaHostRegister(p->base_, kRing * kChunk, cudaHostRegisterPortable) == cudaSuccess;
    if (!p->pinned_) {
      (void)cudaGetLastError();
      return nullptr;
    }
    cpu_set_t cpus;
    const int n = sched_getaffinity(0, sizeof cpus, &cpus) == 0 ? CPU_COUNT(&cpus) : 1;
    try {  // nothing is thrown through the C interface: fewer threads, the caller writes the rest
      for (int k = 0; k < std::min(kMaxThreads, n - 1); ++k) p->threads_.emplace_back([q = p.get()] { q->work(); });
    } catch (...) {
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
    if (pinned_) cudaHostUnregister(base_);
    if (map_) munmap(map_, kMapped);
  }

  cudaError_t copy(char* dst, const char* src, size_t bytes, int device, cudaStream_t stream)
  {
    if (device != events_device_) {  // events belong to a device
      drop_events();
      unsigned flags = 0;  // the caller waits as it has asked to wait for this device
      if (cudaGetDeviceFlags(&flags) != cudaSuccess) (void)cudaGetLastError();
      const bool sleep = (flags & cudaDeviceScheduleMask) == cudaDeviceScheduleBlockingSync;
      for (cudaEvent_t& ev : events_) {
        const cudaError_t e =
          cudaEventCreateWithFlags(&ev, cudaEventDisableTiming | (sleep ? cudaEventBlockingSync : 0));
        if (e != cudaSuccess) {
          drop_events();
          return e;
        }
      }
      events_device_ = device;
    }
    const size_t chunks = (bytes + kChunk - 1) / kChunk;
    size_t issued = 0;
    cudaError_t e = cudaSuccess;
    std::unique_lock<std::mutex> lock(mutex_);
    dst_ = dst;
    bytes_ = bytes;
    taken_ = 0;
    landed_ = 0;
    written_ = 0;
    for (size_t& l : left_) l = 0;
    while (landed_ < chunks && e == cudaSuccess) {
      const size_t b = issued % kRing;
      const bool issue = issued < chunks && issued < landed_ + kRing && left_[b] == issued / kRing;
      if (landed_ < issued) {
        // handed out as soon as it is there, also between two transfers' issues
        const cudaEvent_t ev = events_[landed_ % kRing];
        lock.unlock();
        const cudaError_t there = issue ? cudaEventQuery(ev) : cudaEventSynchronize(ev);
        if (there == cudaErrorNotReady) (void)cudaGetLastError();
        lock.lock();
        if (there == cudaSuccess) {
          if (++landed_ == 1) wake_.notify_all();
          else wake_.notify_one();
          continue;
        }
        if (there != cudaErrorNotReady) {
          e = there;
          continue;
        }
      }
      if (issue) {
        const size_t at = issued++ * kChunk;
        lock.unlock();
        e = cudaMemcpyAsync(base_ + b * kChunk, src + at, std::min(kChunk, bytes - at), cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaEventRecord(events_[b], stream);
        lock.lock();
      } else if (!write_one(lock)) {
        const size_t seen = written_;
        wait(lock, freed_, [&] { return written_ != seen; });
      }
    }
    while (write_one(lock)) {}
    wait(lock, freed_, [&] { return written_ == landed_; });
    if (e != cudaSuccess) {  // no transfer may reach the ring after the copy
      lock.unlock();
      cudaStreamSynchronize(stream);
    }
    return e;
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

  // waits for `there` (atomics only): looks for a while, then sleeps
  template <class F>
  static void wait(std::unique_lock<std::mutex>& lock, std::condition_variable& cv, F&& there)
  {
    if (there()) return;
    lock.unlock();
    const auto until = std::chrono::steady_clock::now() + kLook;
    while (!there() && std::chrono::steady_clock::now() < until) std::this_thread::yield();
    lock.lock();
    cv.wait(lock, there);
  }

  // writes out the next chunk that has landed; false when there is none
  bool write_one(std::unique_lock<std::mutex>& lock)
  {
    if (taken_ == landed_) return false;
    const size_t i = taken_++, at = i * kChunk;
    lock.unlock();
    std::memcpy(dst_ + at, base_ + (i % kRing) * kChunk, std::min(kChunk, bytes_ - at));
    lock.lock();
    ++left_[i % kRing];
    ++written_;
    return true;
  }

  void work()
  {
    (void)pthread_setname_np(pthread_self(), "olb-copy");
    std::unique_lock<std::mutex> lock(mutex_);
    while (!quit_) {
      if (write_one(lock)) {
        freed_.notify_one();
        continue;
      }
      wait(lock, wake_, [&] { return quit_ || taken_ != landed_; });
    }
  }

  void* map_ = nullptr;
  char* base_ = nullptr;  // in map_, on a huge page
  bool pinned_ = false;
  std::vector<std::thread> threads_;
  std::mutex mutex_;
  std::condition_variable wake_, freed_;  // chunks to write; a chunk written
  std::atomic<bool> quit_{false};
  cudaEvent_t events_[kRing] = {};
  int events_device_ = -1;
  // the current copy (mutex_; the atomics are also looked at without it)
  char* dst_ = nullptr;
  size_t bytes_ = 0;
  size_t left_[kRing] = {};                                  // chunks that have left each buffer
  std::atomic<size_t> landed_{0}, taken_{0}, written_{0};  // chunks in the ring so far, taken by a thread, written out
};

// holders, the pool and its use; never destroyed (a handle leaked at exit
// leaves threads that wait, which the exit ends)
struct Shared {
  std::mutex mutex;         // holds, direct, pool
  std::mutex in_use;        // one copy at a time
  int holds = 0;
  size_t direct = 0;        // bytes that could have been staged, since the first of the holders
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
  if (--shared().holds == 0) {
    gone = std::move(shared().pool);
    shared().direct = 0;
  }
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
    if (!s.pool && (s.direct += bytes) >= kRingFrom) s.pool = Pool::make();
    pool = s.pool.get();
  }
  if (!pool) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream);
  return pool->copy(static_cast<char*>(dst), static_cast<const char*>(src), bytes, device, stream);
}

} // namespace olb_b200
