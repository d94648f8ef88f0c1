// host_copy.hpp -- device-to-host copies into pageable memory through a ring of
// pinned pieces and a few copying threads.
//
// A device-to-host copy into pageable memory is staged by the driver on the
// calling thread: 12 GB/s and nothing else overlaps it (5.2 MB: 439 us against
// 105 us into pinned memory).  Here the copy engine fills 512-KiB pinned pieces
// back to back while up to four threads move the finished ones to the
// destination.  The ring (8 MiB), its events and the threads belong to one
// context, are made on its first large pageable download and end with it; the
// context's lock admits one caller at a time.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <condition_variable>
#include <cstring>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace sfntt {

class HostCopier {
 public:
  static constexpr size_t kPiece = (size_t)512 << 10;
  static constexpr int kSlots = 16;

  // nullptr where the ring or the threads cannot be had: the caller then copies directly.
  static std::unique_ptr<HostCopier> create(int device) {
    std::unique_ptr<HostCopier> c;
    try {
      c.reset(new HostCopier(device));
      if (cudaHostAlloc(reinterpret_cast<void**>(&c->ring_), kPiece * kSlots, cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
      }
      for (int i = 0; i < kSlots; ++i)
        if (cudaEventCreateWithFlags(&c->ev_[i], cudaEventDisableTiming) != cudaSuccess) {
          cudaGetLastError();
          return nullptr;
        }
      const unsigned hc = std::thread::hardware_concurrency();
      const unsigned n = std::max(1u, std::min(4u, hc / 2));
      for (unsigned i = 0; i < n; ++i) c->threads_.emplace_back([p = c.get()] { p->work(); });
    } catch (...) {  // no memory, or not every thread
      if (!c || c->threads_.empty()) return nullptr;
    }
    return c;
  }

  ~HostCopier() {
    {
      std::lock_guard<std::mutex> lk(mu_);
      stop_ = true;
    }
    cv_job_.notify_all();
    for (std::thread& t : threads_) t.join();
    for (cudaEvent_t e : ev_)
      if (e) cudaEventDestroy(e);
    if (ring_) cudaFreeHost(ring_);
  }

  // Queues the copy of `bytes` from device memory to dst, behind the work on s.
  // Blocks only while every piece of the ring is in use.
  cudaError_t download(void* dst, const void* src, size_t bytes, cudaStream_t s) {
    for (size_t at = 0; at < bytes; at += kPiece) {
      const size_t len = std::min(kPiece, bytes - at);
      const int slot = next_;
      next_ = (next_ + 1) % kSlots;
      {
        std::unique_lock<std::mutex> lk(mu_);
        cv_free_.wait(lk, [&] { return !busy_[slot]; });
        if (err_ != cudaSuccess) return err_;
        busy_[slot] = true;
      }
      cudaError_t e = cudaMemcpyAsync(ring_ + (size_t)slot * kPiece, static_cast<const char*>(src) + at, len,
                                      cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaEventRecord(ev_[slot], s);
      if (e != cudaSuccess) {
        std::lock_guard<std::mutex> lk(mu_);
        busy_[slot] = false;
        return e;
      }
      {
        std::lock_guard<std::mutex> lk(mu_);
        jobs_[(head_ + queued_++) % kSlots] = {slot, static_cast<char*>(dst) + at, len};  // one per busy piece at most
      }
      cv_job_.notify_one();
    }
    return cudaSuccess;
  }

  // Waits until every queued piece has reached its destination.
  cudaError_t finish() {
    std::unique_lock<std::mutex> lk(mu_);
    cv_free_.wait(lk, [&] { return queued_ == 0 && std::none_of(busy_, busy_ + kSlots, [](bool b) { return b; }); });
    const cudaError_t e = err_;
    err_ = cudaSuccess;
    return e;
  }

 private:
  struct Job { int slot; char* dst; size_t len; };

  explicit HostCopier(int device) : device_(device) {}

  void work() {
    cudaSetDevice(device_);
    std::unique_lock<std::mutex> lk(mu_);
    for (;;) {
      cv_job_.wait(lk, [&] { return stop_ || queued_ > 0; });
      if (queued_ == 0) return;
      const Job j = jobs_[head_];
      head_ = (head_ + 1) % kSlots;
      --queued_;
      lk.unlock();
      const cudaError_t e = cudaEventSynchronize(ev_[j.slot]);
      if (e == cudaSuccess) std::memcpy(j.dst, ring_ + (size_t)j.slot * kPiece, j.len);
      lk.lock();
      if (e != cudaSuccess && err_ == cudaSuccess) err_ = e;
      busy_[j.slot] = false;
      cv_free_.notify_all();
    }
  }

  int device_;
  char* ring_ = nullptr;
  cudaEvent_t ev_[kSlots] = {};
  bool busy_[kSlots] = {};
  int next_ = 0;
  std::mutex mu_;
  std::condition_variable cv_job_, cv_free_;
  Job jobs_[kSlots] = {};  // first in, first out
  int head_ = 0, queued_ = 0;
  std::vector<std::thread> threads_;
  cudaError_t err_ = cudaSuccess;
  bool stop_ = false;
};

}  // namespace sfntt
