// The tile kernels whose waits are their warps' own, one CTA on host threads: a
// copy or an arrival that never lands must end the CTA after one wait that runs
// out per thread, with the error flag set and nothing written after it.
#include "cta.hpp"

#include <cstdio>

#include "tile_warp.cuh"

using namespace sfntt;

namespace {

int failures = 0;
void check(bool ok, const char* what, const char* where) {
  if (!ok) {
    ++failures;
    std::printf("FAILED %s: %s\n", where, what);
  }
}
// A loaded host may be slow to schedule the threads: where nothing is lost no wait may run out.
void patience(bool lost) { cta::limit = std::chrono::milliseconds(lost ? 1000 : 60000); }
int most_expired(int threads) { return *std::max_element(cta::expired.begin(), cta::expired.begin() + threads); }

std::vector<uint2> table(size_t n) { return std::vector<uint2>(n, make_uint2(1, 2)); }

// M31 top pass: 13 bits of positions below the 8 layers, one tile of 12 per column.
void warp_pass(int lose, const char* where) {
  static int err;
  err = 0;
  const auto tw = table(1u << 13);
  CUtensorMap map{};
  TmaArgs a{};
  a.tw = tw.data();
  a.log_n = 13;
  a.lo = 5;
  a.batch = a.ntiles = 12;
  a.err = &err;
  patience(lose >= 0);
  cta::lose_load = lose;
  cta::lose_arrival = nullptr;
  cta::run(wt::kThreads, [&] { WPass<M31, true>::run(&map, &map, a); });
  const int stored = (int)cta::stores.size();
  check(stored == (lose < 0 ? 12 : lose), "tiles stored: those before the lost one", where);
  for (int i = 0; i < stored; ++i) check(cta::stores[i][4] == i, "tiles stored in order", where);
  check(err == (lose >= 0), "error flag", where);
  check(most_expired(32 * wt::kWarps) == (lose >= 0), "one wait that runs out per compute thread", where);
  check(cta::expired[32 * wt::kWarps] <= 1 + wt::kRing, "the mover: one wait, then its loads in flight", where);
}

// M31 expansion of 6 tiles into 2^log_q blocks each.  lose: a tile's load; lose_free:
// the mover's report that a buffer's store has read it (index among its reports).
void warp_expand(uint32_t log_q, int lose, int lose_free, const char* where) {
  static int err;
  err = 0;
  const auto tw = table(1u << 13), tf = table(1u << 15);
  CUtensorMap map{};
  TmaArgs a{};
  a.tw = tw.data();
  a.tw_fwd = tf.data();
  a.log_n = 13;
  a.lo = 5;
  a.batch = a.ntiles = 6;
  a.log_q = log_q;
  a.scale_w = 1;
  a.scale_ws = 2;
  a.err = &err;
  const int nq = 1 << log_q, blocks = 6 * nq;
  int reports = 0;
  patience(lose >= 0 || lose_free >= 0);
  cta::lose_load = lose;
  cta::lose_arrival = [&](uint32_t tid, int) { return tid == 32u * wt::kWarps && reports++ == lose_free; };
  cta::run(wt::kThreads, [&] { WExpandM31::run(&map, &map, a); });
  const int stored = (int)cta::stores.size();
  if (lose < 0 && lose_free < 0) check(stored == blocks, "every block stored", where);
  if (lose >= 0) check(stored == lose * nq, "blocks stored: those of the tiles before the lost one", where);
  // buffer k's next block is k + 3; a tile's first block does not wait for the report
  if (lose_free >= 0) check(stored <= lose_free + 3, "no block through a buffer that was not given back", where);
  for (int i = 0; i < stored; ++i)
    check(cta::stores[i][4] == i / nq && cta::stores[i][3] == i % nq, "blocks stored in order", where);
  const bool lost = lose >= 0 || lose_free >= 0;
  check(err == (int)lost, "error flag", where);
  check(most_expired(32 * wt::kWarps) == (int)lost, "one wait that runs out per compute thread", where);
}

// Two columns at once, 3 pairs of 2^13 points, 8x, in place.  lose: index of the
// warps' "has read" arrivals that is dropped (16 per exchange).
void expand_cols(int lose, const char* where) {
  using X = TExpandCols<BabyBear>;
  static int err;
  err = 0;
  const auto tw = table(1u << 13), tf = table(1u << 16), mul = table(1u << 16);
  const uint32_t n = 1u << 13, nq = 8, cols = 6;
  std::vector<uint32_t> out((size_t)cols * n * nq, 0xABABABABu);
  TmaArgs a{};
  a.tw = tw.data();
  a.tw_fwd = tf.data();
  a.mul = mul.data();
  a.out = out.data();
  a.out_stride = (uint64_t)n * nq;
  a.log_n = 13;
  a.lo = 5;
  a.batch = cols;
  a.log_q = 3;
  a.ntiles = cols / 2;
  a.err = &err;
  patience(lose >= 0);
  cta::lose_load = -1;
  cta::lose_arrival = [&](uint32_t, int i) { return i == lose; };
  cta::run(X::NT, [&] { X::run(a); });
  // blocks of a column whose words were written (the start value stays canonical-free)
  auto written = [&](uint32_t col, uint32_t q) {
    const uint32_t* p = out.data() + ((size_t)col * nq + q) * n;
    return std::any_of(p, p + n, [](uint32_t x) { return x != 0xABABABABu; });
  };
  const int warps = X::NT / 32;
  for (uint32_t col = 0; col < cols; ++col)
    for (uint32_t q = 0; q < nq; ++q) {
      // block q of a pair's column is written after the pair's exchange 1 + q; the
      // arrivals of exchange e are waited for before exchange e + 1 is written
      const int exchange = (int)(col / 2 * (nq + 1) + 1 + q);
      const bool before = lose < 0 || exchange < lose / warps;
      check(written(col, q) == before, before ? "block written" : "nothing written after the lost arrival", where);
    }
  check(err == (lose >= 0), "error flag", where);
  check(most_expired(X::NT) == (lose >= 0), "one wait that runs out per thread", where);
}

}  // namespace

int main() {
  warp_pass(-1, "top pass, nothing lost");
  warp_pass(0, "top pass, first load lost");
  warp_pass(4, "top pass, load 4 lost");
  warp_expand(1, -1, -1, "expansion 2x, nothing lost");
  warp_expand(2, -1, -1, "expansion 4x, nothing lost");
  warp_expand(1, 2, -1, "expansion 2x, load 2 lost");
  warp_expand(2, 1, -1, "expansion 4x, load 1 lost");
  warp_expand(1, -1, 4, "expansion 2x, report 4 lost");
  warp_expand(2, -1, 3, "expansion 4x, report 3 lost");
  expand_cols(-1, "two columns, nothing lost");
  expand_cols(0, "two columns, first arrival lost");
  expand_cols(16 * 5 + 3, "two columns, an arrival of exchange 5 lost");
  if (!failures) std::printf("all ok\n");
  return failures != 0;
}
