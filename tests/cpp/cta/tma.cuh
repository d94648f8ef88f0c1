// Host stand-in for the bulk copies, mbarriers and shared-memory accesses.
#pragma once
#include "cta.hpp"

namespace sfntt {
namespace tma {

inline uint32_t smem_addr(const void* p) {
  return (uint32_t)(reinterpret_cast<const char*>(p) - reinterpret_cast<const char*>(smem_words));
}
inline uint32_t* at(uint32_t a) { return smem_words + a / 4; }
inline uint32_t lds32(uint32_t a) { return *at(a); }
inline uint4 lds128(uint32_t a) { return make_uint4(at(a)[0], at(a)[1], at(a)[2], at(a)[3]); }
inline void sts32(uint32_t a, uint32_t x) { *at(a) = x; }
inline void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  at(a)[0] = x; at(a)[1] = y; at(a)[2] = z; at(a)[3] = w;
}

inline void mbar_init(uint64_t* bar, uint32_t count) {
  std::lock_guard<std::mutex> lk(cta::mu);
  cta::mbars[bar] = {count, count, 0, 0};
}
inline void fence_mbar_init() {}
inline void fence_proxy_async() {}
inline void prefetch_map(const CUtensorMap*) {}
inline void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  std::lock_guard<std::mutex> lk(cta::mu);
  cta::Mbar& b = cta::mbars[bar];
  b.tx += bytes;
  --b.pending;
  cta::settle(b);
}
inline void mbar_arrive(uint64_t* bar) {
  std::lock_guard<std::mutex> lk(cta::mu);
  if (cta::lose_arrival && cta::lose_arrival(threadIdx.x, cta::arrivals++)) return;
  cta::Mbar& b = cta::mbars[bar];
  --b.pending;
  cta::settle(b);
}
inline bool mbar_wait(uint64_t* bar, uint32_t parity, uint64_t) {
  std::unique_lock<std::mutex> lk(cta::mu);
  cta::Mbar& b = cta::mbars[bar];
  if (cta::cv.wait_for(lk, cta::limit, [&] { return b.phase != parity; })) return true;
  ++cta::expired[threadIdx.x];
  return false;
}

// A whole tile of words lands at once (its contents do not matter here).
inline void land(void* dst, uint64_t* bar) {
  std::lock_guard<std::mutex> lk(cta::mu);
  if (cta::loads++ == cta::lose_load) return;
  cta::Mbar& b = cta::mbars[bar];
  std::memset(dst, 0, (size_t)b.tx);
  b.tx = 0;
  cta::settle(b);
}
inline void load_3d(void* dst, const CUtensorMap*, int32_t, int32_t, int32_t, uint64_t* bar) { land(dst, bar); }
inline void load_5d(void* dst, const CUtensorMap*, int32_t, int32_t, int32_t, int32_t, int32_t, uint64_t* bar) {
  land(dst, bar);
}
inline void store_3d(const CUtensorMap*, int32_t c0, int32_t c1, int32_t c2, const void*) {
  std::lock_guard<std::mutex> lk(cta::mu);
  cta::stores.push_back({c0, c1, c2});
}
inline void store_5d(const CUtensorMap*, int32_t c0, int32_t c1, int32_t c2, int32_t c3, int32_t c4, const void*) {
  std::lock_guard<std::mutex> lk(cta::mu);
  cta::stores.push_back({c0, c1, c2, c3, c4});
}
inline void store_bulk(void*, const void*, uint32_t) { std::abort(); }
inline void commit() {}
inline void wait_reads() {}
inline void wait_reads_1() {}
inline void wait_all() {}

}  // namespace tma
}  // namespace sfntt
