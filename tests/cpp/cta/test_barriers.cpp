// Named barriers of kernels that run one network and then the other on a tile with
// no CTA barrier between: an id may stand for one set of threads only, or a warp
// ahead in the second network arrives at a barrier that others of the first still
// wait at.
#include "cta.hpp"

#include <cstdio>
#include <set>

#include "tile_tma.cuh"

using namespace sfntt;

namespace {

int failures = 0;
using Ids = std::map<uint32_t, std::set<uint32_t>>;  // id -> threads that meet there

template <class T, bool DESC>
void exchanges(std::vector<Ids>& out) {
  for (int i = 1; i < T::K; ++i) {
    const int kp = DESC ? T::K - i : i - 1, k = DESC ? T::K - 1 - i : i;
    if (T::xgroups(kp, k) == 0) continue;  // a warp or CTA barrier
    const int wf = T::xfixed_of(kp, k) & T::kWarpBits;
    Ids ids;
    for (uint32_t tid = 0; tid < (uint32_t)T::NT; ++tid) {
      uint32_t id = (uint32_t)T::xbase(i), n = 0;
      for (int bit = 5; bit < 16; ++bit)
        if ((wf >> bit) & 1) id += ((tid >> bit) & 1u) << n++;
      ids[id].insert(tid);
    }
    out.push_back(ids);
  }
}

template <class A, bool AD, class B, bool BD>
void check(const char* what, int P) {
  std::vector<Ids> e;
  exchanges<A, AD>(e);
  exchanges<B, BD>(e);
  for (size_t i = 0; i < e.size(); ++i)
    for (size_t j = 0; j < i; ++j)
      for (auto& [id, threads] : e[i]) {
        auto it = e[j].find(id);
        if (it == e[j].end() || it->second == threads) continue;
        ++failures;
        std::printf("FAILED %s, %d layers: id %u stands for two sets of threads (exchanges %zu and %zu)\n", what, P, id, j, i);
        return;
      }
}

template <class F, int P, int TB>
void both(const char* what) {
  using Inv = TPass<F, false, Kind::C, P, false, false, false, false, TB>;
  using Fwd = TPass<F, true, Kind::C, P, false, false, false, false, TB>;
  check<Inv, false, Fwd, true>(what, P);
  check<Fwd, true, Inv, false>(what, P);
}

template <class F>
void all(const char* what) {
  both<F, 5, 11>(what);
  both<F, 6, 11>(what);
  both<F, 7, 11>(what);
  both<F, 8, 11>(what);
  both<F, 9, 11>(what);
  both<F, 10, 11>(what);
  both<F, 11, 11>(what);
  both<F, 12, 12>(what);
  both<F, 13, 13>(what);
  both<F, 14, 14>(what);
}

}  // namespace

int main() {
  all<BabyBear>("short-column LDE, BabyBear");
  all<M31>("short-column LDE, M31");
  both<BabyBear, 12, 0>("natural-order expansion");
  if (!failures) std::printf("all ok\n");
  return failures != 0;
}
