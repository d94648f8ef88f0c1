// Which buffers the one-launch LDE of short columns takes: its CTAs read and write
// without an order between them, so the input may lie in the output only where each
// column sits in its own output column from the start.
#include <cstdio>

#include "../../small-field-metal-ntt_b200/csrc/context.hpp"

int main() {
  sfntt_ctx& ctx = *new sfntt_ctx;  // no device: kept to the end
  ctx.sm_count = 148;
  alignas(16) static uint32_t words[1];
  uint32_t* out = words;  // addresses only: nothing is read
  int failures = 0;
  auto expect = [&](bool want, const uint32_t* in, uint64_t stride, uint32_t log_n, uint32_t batch, uint32_t added,
                    const char* what) {
    if (sfntt::lde_small_fits(&ctx, in, out, stride, log_n, batch, added) != want) {
      ++failures;
      std::printf("FAILED 2^%u x %u, 2^%u x: %s\n", log_n, batch, added, what);
    }
  };
  for (uint32_t log_n = 5; log_n <= 14; ++log_n)
    for (uint32_t batch : {1u, 3u, 37u})
      for (uint32_t added : {1u, 2u}) {
        const uint64_t n = 1ull << log_n, n_ext = n << added, in_words = batch * n, out_words = batch * n_ext;
        const bool short_col = log_n < 14;
        expect(true, out + out_words, n, log_n, batch, added, "input behind the output");
        expect(true, out - in_words, n, log_n, batch, added, "input before the output");
        expect(short_col, out, n_ext, log_n, batch, added, "columns in their own output columns");
        expect(batch == 1 && short_col, out, n, log_n, batch, added, "dense input at the output's start");
        expect(false, out + n, n, log_n, batch, added, "input in a later block of the output");
        expect(false, out + out_words - in_words, n, log_n, batch, added, "input at the output's end");
        expect(false, out + out_words - 4, n, log_n, batch, added, "input starting in the output's last words");
        expect(false, out - in_words + 4, n, log_n, batch, added, "input ending in the output's first words");
        expect(false, out + n, n_ext, log_n, batch, added, "columns in later blocks of their output columns");
      }
  if (!failures) std::printf("all ok\n");
  return failures != 0;
}
