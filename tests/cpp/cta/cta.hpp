// cta.hpp -- runs one CTA of a tile kernel on host threads, so that a wait that
// runs out can be watched without a GPU.
//
// Included before the kernel headers (copied beside this folder's pdl.cuh and
// tma.cuh, which take the place of the PTX ones).  One host thread per CUDA
// thread; barriers are real barriers, mbarriers count arrivals, and a copy or
// an arrival named in `cta::lose` never lands.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <barrier>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#undef __launch_bounds__
#define __launch_bounds__(...)
#undef __grid_constant__
#define __grid_constant__

using std::min;

namespace cta {

struct Dim { uint32_t x = 0; };
inline thread_local Dim thread_idx;
inline Dim block_idx, grid_dim{1};

// A barrier whose members may leave (a thread that returns).
struct Group {
  std::barrier<> bar;
  std::atomic<int> votes{0};
  explicit Group(int n) : bar(n) {}
  void sync() { bar.arrive_and_wait(); }
  bool any(bool x) {
    if (x) votes.fetch_add(1);
    bar.arrive_and_wait();
    const bool r = votes.load() != 0;
    bar.arrive_and_wait();
    votes.store(0);
    bar.arrive_and_wait();
    return r;
  }
};
inline std::unique_ptr<Group> block;
inline std::vector<std::unique_ptr<Group>> warps;
inline Group& warp() { return *warps[thread_idx.x / 32]; }

struct Mbar { uint32_t count = 0, pending = 0, phase = 0; int64_t tx = 0; };
inline std::mutex mu;
inline std::condition_variable cv;
inline std::map<const void*, Mbar> mbars;
inline std::vector<int> expired;                      // waits that ran out, per thread
inline std::chrono::milliseconds limit{1000};         // for every bounded wait
inline int loads = 0, arrivals = 0;
inline int lose_load = -1;                            // index of the load that never lands
inline std::function<bool(uint32_t, int)> lose_arrival;  // (thread, index among all plain arrivals)
inline std::vector<std::vector<int32_t>> stores;      // coordinates, in order

inline void settle(Mbar& b) {
  if (b.pending == 0 && b.tx == 0) {
    b.phase ^= 1u;
    b.pending = b.count;
    cv.notify_all();
  }
}

template <class Fn>
void run(int threads, Fn kernel) {
  block = std::make_unique<Group>(threads);
  warps.clear();
  for (int w = 0; w < threads / 32; ++w) warps.push_back(std::make_unique<Group>(32));
  mbars.clear();
  stores.clear();
  loads = arrivals = 0;
  expired.assign(threads, 0);
  std::vector<std::thread> ts;
  for (int t = 0; t < threads; ++t)
    ts.emplace_back([&, t] {
      thread_idx.x = (uint32_t)t;
      kernel();
      warp().bar.arrive_and_drop();
      block->bar.arrive_and_drop();
    });
  for (auto& t : ts) t.join();
}

}  // namespace cta

#define threadIdx cta::thread_idx
#define blockIdx cta::block_idx
#define gridDim cta::grid_dim

inline void __syncthreads() { cta::block->sync(); }
inline int __syncthreads_or(int x) { return cta::block->any(x != 0); }
inline void __syncwarp(unsigned = ~0u) { cta::warp().sync(); }
inline int __all_sync(unsigned, int x) { return !cta::warp().any(x == 0); }
inline unsigned __shfl_xor_sync(unsigned, unsigned, int) { std::abort(); }
inline uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
inline int __clz(uint32_t x) { return x ? __builtin_clz(x) : 32; }
template <class T>
inline T __ldg(const T* p) { return *p; }
inline int atomicExch(int* p, int v) { return __atomic_exchange_n(p, v, __ATOMIC_SEQ_CST); }

namespace sfntt {
alignas(1024) inline uint32_t smem_words[232448 / 4];
}
