// Copies from ordinary (pageable) host memory to the device.
//
// cudaMemcpyAsync stages pageable memory through the driver on one thread: 17 GB/s for a few megabytes and 10 GB/s for tens,
// against 54 GB/s from pinned memory.  Here the calling thread and three helpers copy 512 KB pieces into a ring of pinned
// memory while the copy engine drains it.  The ring (8 MB) and the helpers belong to one device's model and go with it; the
// calls on a device are serialised by the library's lock, and the helpers touch a caller's memory only while its call runs.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>

namespace nncv_b200 {

class HostCopier {
 public:
  // Below this the driver's own staging is faster (4.8 MB: 265 us against 544; 38 MB: 3024 against 1717).
  static constexpr size_t kWorthIt = 16 << 20;
  HostCopier() = default;
  HostCopier(const HostCopier&) = delete;
  HostCopier& operator=(const HostCopier&) = delete;
  ~HostCopier() {   // no copy of this object is in flight
    {
      std::lock_guard<std::mutex> lk(mu_);
      quit_ = true;
      cv_.notify_all();
    }
    for (auto& t : helpers_)
      if (t.joinable()) t.join();
    for (auto& d : done_)
      if (d) cudaEventDestroy(d);
    if (ring_) cudaFreeHost(ring_);
  }
  // Enqueues the copy on `st`; returns when every byte of src has been read.
  cudaError_t copy(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    cudaError_t e = start();
    if (e != cudaSuccess) return e;
    Job& j = job_;
    j.src = static_cast<const char*>(src);
    j.bytes = bytes;
    j.pieces = (long)((bytes + kPiece - 1) / kPiece);
    j.base = seq_;
    j.allowed.store(0);
    j.next.store(0);
    {
      std::lock_guard<std::mutex> lk(mu_);
      ++generation_;
      open_ = true;
      cv_.notify_all();
    }
    long issued = 0;
    while (issued < j.pieces) {
      const long a = j.allowed.load(std::memory_order_relaxed);
      if (a < j.pieces && a < issued + kSlots) {   // a free slot: its last copy has left it
        const cudaError_t q = cudaEventQuery(done_[(j.base + a) % kSlots]);
        if (q == cudaSuccess) {
          ready_[(j.base + a) % kSlots].store(0, std::memory_order_relaxed);
          j.allowed.store(a + 1, std::memory_order_release);
        } else if (q != cudaErrorNotReady) {
          e = q;
          break;
        }
      }
      const int slot = (int)((j.base + issued) % kSlots);
      if (issued < j.allowed.load(std::memory_order_relaxed) && ready_[slot].load(std::memory_order_acquire)) {
        const size_t off = (size_t)issued * kPiece, n = bytes - off < kPiece ? bytes - off : kPiece;
        if ((e = cudaMemcpyAsync(static_cast<char*>(dst) + off, ring_ + (size_t)slot * kPiece, n, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
            (e = cudaEventRecord(done_[slot], st)) != cudaSuccess)
          break;
        ++issued;
        continue;
      }
      take_one(j);
    }
    seq_ = (j.base + j.pieces) % kSlots;
    j.next.store(j.pieces);                        // no helper starts another piece
    {
      std::unique_lock<std::mutex> lk(mu_);
      open_ = false;                               // a helper that wakes only now finds nothing to do and is not waited for
      idle_.wait(lk, [&] { return busy_ == 0; });
    }
    return e;
  }

 private:
  static constexpr size_t kPiece = 512 << 10;
  static constexpr int kSlots = 16, kHelpers = 3;
  struct Job {
    const char* src = nullptr;
    size_t bytes = 0;
    long pieces = 0, base = 0;
    std::atomic<long> next{0}, allowed{0};
  };
  // Copies the next piece whose slot is free, if there is one.
  bool take_one(Job& j) {
    long i = j.next.load(std::memory_order_relaxed);
    if (i >= j.pieces || i >= j.allowed.load(std::memory_order_acquire)) return false;
    if (!j.next.compare_exchange_strong(i, i + 1)) return false;
    const size_t off = (size_t)i * kPiece, n = j.bytes - off < kPiece ? j.bytes - off : kPiece;
    const int slot = (int)((j.base + i) % kSlots);
    memcpy(ring_ + (size_t)slot * kPiece, j.src + off, n);
    ready_[slot].store(1, std::memory_order_release);
    return true;
  }
  cudaError_t start() {
    if (ring_) return cudaSuccess;
    char* r = nullptr;
    cudaError_t e = cudaHostAlloc((void**)&r, kSlots * kPiece, cudaHostAllocDefault);
    if (e != cudaSuccess) return e;
    for (auto& d : done_)
      if (!d && (e = cudaEventCreateWithFlags(&d, cudaEventDisableTiming)) != cudaSuccess) {
        cudaFreeHost(r);
        return e;
      }
    ring_ = r;
    try {
      for (auto& t : helpers_) t = std::thread([this] { help(); });
    } catch (const std::system_error&) {   // no more threads to be had: those there are, at least the caller's, do the copying
    }
    return cudaSuccess;
  }
  void help() {
    unsigned seen = 0;
    std::unique_lock<std::mutex> lk(mu_);
    for (;;) {
      cv_.wait(lk, [&] { return generation_ != seen || quit_; });
      if (quit_) return;
      seen = generation_;
      if (!open_) continue;
      ++busy_;
      lk.unlock();
      while (job_.next.load(std::memory_order_relaxed) < job_.pieces)
        if (!take_one(job_)) std::this_thread::yield();
      lk.lock();
      if (--busy_ == 0) idle_.notify_all();
    }
  }
  Job job_;
  char* ring_ = nullptr;
  cudaEvent_t done_[kSlots] = {};
  std::atomic<int> ready_[kSlots] = {};
  long seq_ = 0;
  std::mutex mu_;
  std::condition_variable cv_, idle_;
  unsigned generation_ = 0;
  int busy_ = 0;        // helpers at work
  bool open_ = false, quit_ = false;
  std::thread helpers_[kHelpers];
};

}  // namespace nncv_b200
