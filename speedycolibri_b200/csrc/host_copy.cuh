// Copies between the caller's pageable memory and the device for the host-pointer calls.
//
// The driver copies pageable memory through staging buffers of its own, one thread, before and after the transfer:
// 1.3 MB took 92 us to the device and 103 back where the link needs 24.  Here a ring of page-locked chunks
// (4 MB a device) stands between: the calling thread and up to three helpers copy chunks while kernels move others over the link, which
// also convert what has to be converted.  A chunk that has arrived is announced by a word in the same memory:
// with a copy command and an event for each chunk the same ring was no faster than the driver (90 + 95 us).
// Memory that is page-locked already, and less than kDirectBytes, goes as it is.
#pragma once
#include <cuda.h>
#include <unistd.h>

#include <atomic>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "internal.cuh"

namespace colib_host {

constexpr size_t kChunk = colib::HOST_CHUNK;
constexpr int kHalf = 32;                    // chunks of one half of the ring; a batch fills a half
// Expert group calls of 8 experts, H 2048, us with the driver's copies and with the ring: 64 KB of rows 82 / 78, 96 KB 91 / 84, 128 KB
// 94 / 87, 192 KB 103 / 92, 256 KB 113 / 97, 1 MB 250 / 168, 4 MB 580 / 367, 16 MB 1900 / 1010, 256 MB 79 400 / 35 400; block calls
// with 32 KB of rows 63 / 62, 64 KB 67 / 66, 96 KB 94 / 85.
constexpr size_t kDirectBytes = 64 * 1024;

// One batch of chunks: chunk i may be copied once i < ready, and is when done[i].
struct CopyBatch {
  char *dst;
  const char *src;
  size_t bytes;
  int n;
  std::atomic<int> next{0}, ready{0};
  std::atomic<bool> done[kHalf] = {};
  bool copy_one() {  // false: nothing to do at the moment
    int i = next.load(std::memory_order_relaxed);
    do {
      if (i >= ready.load(std::memory_order_acquire)) return false;
    } while (!next.compare_exchange_weak(i, i + 1, std::memory_order_relaxed));
    const size_t at = (size_t)i * kChunk;
    memcpy(dst + at, src + at, bytes - at < kChunk ? bytes - at : kChunk);
    done[i].store(true, std::memory_order_release);
    return true;
  }
};

// The helping threads of the process: started by the first call that can use them, asleep between calls, joined
// by the library's shutdown or the end of the process.  One call has them at a time; another works alone.
// A forked child has this object, in whatever state, and none of the threads: there it is not touched.
class CopyPool {
 public:
  bool begin() {
    if (forked() || !owner_.try_lock()) return false;
    std::lock_guard<std::mutex> lk(mu_);
    if (threads_.empty()) {
      pid_.store(getpid());
      const unsigned cores = std::thread::hardware_concurrency();
      const int want = cores >= 8 ? 3 : cores >= 4 ? 1 : 0;
      stop_ = false;
      try {
        for (int i = 0; i < want; ++i) threads_.emplace_back([this] { work(); });
      } catch (...) {  // as many as there are
      }
    }
    active_.store(true, std::memory_order_release);
    ++session_;
    cv_.notify_all();
    return true;
  }
  void end() {
    active_.store(false, std::memory_order_release);
    owner_.unlock();
  }
  void offer(CopyBatch *b) { batch_.store(b); }
  void withdraw() {  // returns when no thread looks at the batch any more
    batch_.store(nullptr);
    while (users_.load() != 0) std::this_thread::yield();
  }
  bool stop() {  // false: nothing done, in a forked child
    if (forked()) return false;
    std::lock_guard<std::mutex> own(owner_);
    {
      std::lock_guard<std::mutex> lk(mu_);
      stop_ = true;
      cv_.notify_all();
    }
    for (auto &t : threads_) t.join();
    threads_.clear();
    return true;
  }
  static void pause() {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#endif
  }

 private:
  bool forked() const {
    const pid_t p = pid_.load();
    return p != 0 && p != getpid();
  }
  void work() {
    uint64_t seen = 0;
    for (;;) {
      {
        std::unique_lock<std::mutex> lk(mu_);
        cv_.wait(lk, [&] { return stop_ || session_ != seen; });
        if (stop_) return;
        seen = session_;
      }
      // awake for the length of a call, whose two copies are some hundred microseconds apart; from a call that takes
      // milliseconds between them the thread goes back to sleep
      for (int idle = 0; idle < 10000 && active_.load(std::memory_order_acquire);) {
        users_.fetch_add(1);
        CopyBatch *b = batch_.load();
        const bool did = b && b->copy_one();
        users_.fetch_sub(1);
        idle = did ? 0 : idle + 1;
        if (!did)
          for (int i = 0; i < 16; ++i) pause();
      }
    }
  }
  std::atomic<pid_t> pid_{0};  // whose threads they are
  std::mutex owner_, mu_;
  std::condition_variable cv_;
  std::vector<std::thread> threads_;
  uint64_t session_ = 0;  // under mu_
  bool stop_ = false;     // under mu_
  std::atomic<bool> active_{false};
  std::atomic<CopyBatch *> batch_{nullptr};
  std::atomic<int> users_{0};
};
// The library's pool.  (Members of a pool whose threads are gone are not destroyed either: the condition variable would
// wait for its sleepers.)
struct LibraryPool {
  CopyPool *const pool = new CopyPool;
  ~LibraryPool() {
    if (pool->stop()) delete pool;
  }
};

// The ring of one device; used by one call at a time (the device's mutex is held).
struct HostRing {
  char *mem = nullptr;                    // two halves of chunks
  volatile uint32_t *arrived = nullptr;   // behind them: a word a chunk, the batch that it holds
  volatile int32_t *status = nullptr;     // and one for the status word of a call's kernels
  cudaEvent_t read[2] = {};               // the device has read a half
  uint32_t batch = 0;
  bool tried = false;
  bool ready() {
    if (tried) return mem != nullptr;
    tried = true;
    void *p = nullptr;
    const size_t chunks = 2 * kHalf;
    if (cudaHostAlloc(&p, chunks * kChunk + (chunks + 1) * sizeof(uint32_t), cudaHostAllocDefault) != cudaSuccess || !p) {
      cudaGetLastError();
      return false;
    }
    for (cudaEvent_t &e : read)
      if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        cudaGetLastError();
        mem = (char *)p;
        release();
        tried = true;
        return false;
      }
    memset((char *)p + chunks * kChunk, 0, (chunks + 1) * sizeof(uint32_t));
    arrived = (volatile uint32_t *)((char *)p + chunks * kChunk);
    status = (volatile int32_t *)(arrived + chunks);
    mem = (char *)p;
    return true;
  }
  void release() {
    for (cudaEvent_t &e : read) {
      if (e) cudaEventDestroy(e);
      e = nullptr;
    }
    if (mem) cudaFreeHost(mem);
    mem = nullptr;
    tried = false;
  }
};

inline bool pointer_attribute(void *value, CUpointer_attribute which, CUdeviceptr at) {
  using Fn = CUresult (*)(void *, CUpointer_attribute, CUdeviceptr);
  static const Fn attribute = [] {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuPointerGetAttribute", &fn, cudaEnableDefault, &found) == cudaSuccess && found == cudaDriverEntryPointSuccess)
      return reinterpret_cast<Fn>(fn);
    cudaGetLastError();
    return Fn(nullptr);
  }();
  return attribute && attribute(value, which, at) == CUDA_SUCCESS;
}

// Whether all of `bytes` at `host`, whose attributes are `a`, is of one page-locked allocation or registration.
inline bool page_locked(const cudaPointerAttributes &a, size_t bytes) {
  if (a.type != cudaMemoryTypeHost || !a.devicePointer) return false;
  CUdeviceptr start = 0;
  size_t size = 0;
  const CUdeviceptr at = reinterpret_cast<CUdeviceptr>(a.devicePointer);
  if (!pointer_attribute(&start, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, at) || !pointer_attribute(&size, CU_POINTER_ATTRIBUTE_RANGE_SIZE, at)) return false;
  return at >= start && at - start <= size && bytes <= size - (at - start);
}

// The device's address of page-locked memory that kernels may write directly, null for any other (also for a buffer of
// which only some pages are registered, and for one that is registered for the device to read only).
inline void *mapped_host(void *host, size_t bytes) {
  cudaPointerAttributes a = {};
  if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  unsigned long long access = 0;
  if (!page_locked(a, bytes) || !pointer_attribute(&access, CU_POINTER_ATTRIBUTE_ACCESS_FLAGS, reinterpret_cast<CUdeviceptr>(a.devicePointer))) return nullptr;
  return (access & CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READWRITE) == CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READWRITE ? a.devicePointer : nullptr;
}

// Of one host-pointer call: its copies to and from the device on stream `st`.  Sizes are multiples of 16 bytes.
class HostCopies {
 public:
  HostCopies(HostRing &ring, CopyPool &pool, cudaStream_t st) : ring_(ring), pool_(pool), st_(st) {}
  ~HostCopies() {
    if (helped_) pool_.end();
  }
  // Whether `bytes` at `host` go through the ring; wakes the helpers if they do.
  bool staged(const void *host, size_t bytes) {
    if (bytes < kDirectBytes || bytes % 16 || !ring_.ready()) return false;
    cudaPointerAttributes a = {};
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess)
      cudaGetLastError();
    else if (a.type != cudaMemoryTypeUnregistered && (a.type != cudaMemoryTypeHost || page_locked(a, bytes)))
      return false;
    if (!helped_) helped_ = pool_.begin();
    return true;
  }
  // `src` has been read when this returns.  to_f16: `src` holds f32, `dst` their f16 (launch_f32_to_f16).
  bool upload(void *dst, const void *src, size_t bytes, bool to_f16, const char *what) {
    for (size_t base = 0, b = 0; base < bytes; base += kHalf * kChunk, ++b) {
      const int half = (int)(b & 1);
      if (b >= 2 && !coli_cuda_check(cudaEventSynchronize(ring_.read[half]), what)) return false;
      CopyBatch c;
      fill(c, ring_.mem + half * kHalf * kChunk, (const char *)src + base, bytes - base);
      c.ready.store(c.n);
      if (helped_) pool_.offer(&c);
      for (int copied = 0; copied < c.n;) {
        if (!c.copy_one()) CopyPool::pause();
        while (copied < c.n && c.done[copied].load(std::memory_order_acquire)) ++copied;
      }
      if (helped_) pool_.withdraw();
      if (!colib::launch_from_host((char *)dst + (to_f16 ? base / 2 : base), c.dst, c.bytes, to_f16, st_) ||
          !coli_cuda_check(cudaEventRecord(ring_.read[half], st_), what))
        return false;
    }
    return true;
  }
  // `dst` is written when this returns.  from_bf16: `src` holds bf16, `dst` is given f32; `bytes` are those of `dst`.
  bool download(void *dst, const void *src, size_t bytes, bool from_bf16, const char *what) {
    auto send = [&](size_t b) {  // queue batch b, if there is one, into its half
      const size_t base = b * kHalf * kChunk;
      if (base >= bytes) return true;
      const size_t n = bytes - base < kHalf * kChunk ? bytes - base : kHalf * kChunk;
      const int half = (int)(b & 1);
      return colib::launch_to_host(ring_.mem + half * kHalf * kChunk, (const char *)src + (from_bf16 ? base / 2 : base), n, from_bf16,
                                   (uint32_t *)ring_.arrived + half * kHalf, first_batch_ + (uint32_t)b, st_) != 0;
    };
    first_batch_ = ring_.batch + 1;
    ring_.batch += (uint32_t)((bytes + kHalf * kChunk - 1) / (kHalf * kChunk));
    if (!send(0) || !send(1)) return false;
    for (size_t base = 0, b = 0; base < bytes; base += kHalf * kChunk, ++b) {
      const int half = (int)(b & 1);
      volatile uint32_t *arrived = ring_.arrived + half * kHalf;
      CopyBatch c;
      fill(c, (char *)dst + base, ring_.mem + half * kHalf * kChunk, bytes - base);
      if (helped_) pool_.offer(&c);
      cudaError_t e = cudaErrorNotReady;
      int here = 0, copied = 0;
      for (uint32_t polls = 0; copied < c.n;) {
        const int before = here;
        while (here < c.n && arrived[here] == first_batch_ + (uint32_t)b) ++here;
        if (here > before) {
          c.ready.store(here, std::memory_order_release);
        } else if (here < c.n && (++polls & 0xfffu) == 0) {  // has the stream failed, or ended without the chunk?
          e = cudaStreamQuery(st_);
          if (e != cudaErrorNotReady && arrived[here] != first_batch_ + (uint32_t)b) break;
          e = cudaErrorNotReady;
        }
        if (!c.copy_one()) CopyPool::pause();
        while (copied < c.n && c.done[copied].load(std::memory_order_acquire)) ++copied;
      }
      if (helped_) pool_.withdraw();
      cudaGetLastError();  // a query that came too early is no error
      if (copied < c.n) return coli_cuda_check(e == cudaSuccess ? cudaErrorUnknown : e, what);
      if (!send(b + 2)) return false;
    }
    return true;
  }

 private:
  static void fill(CopyBatch &c, char *dst, const char *src, size_t left) {
    c.dst = dst, c.src = src;
    c.bytes = left < kHalf * kChunk ? left : kHalf * kChunk;
    c.n = (int)((c.bytes + kChunk - 1) / kChunk);
  }
  HostRing &ring_;
  CopyPool &pool_;
  cudaStream_t st_;
  bool helped_ = false;
  uint32_t first_batch_ = 0;
};

}  // namespace colib_host
