// Which strided passes are launched early: short ones only as grids of one round.
#include <cstdio>

#include "../../small-field-metal-ntt_b200/csrc/pdl.cuh"

int main() {
  using sfntt::pdl_fits_strided;
  int failures = 0;
  auto expect = [&](bool want, int layers, unsigned ctas, unsigned tiles, unsigned log_n, const char* what) {
    if (pdl_fits_strided(layers, ctas, tiles, log_n) != want) {
      ++failures;
      std::printf("FAILED %d layers, %u CTAs, %u tiles: %s\n", layers, ctas, tiles, what);
    }
  };
  for (int layers = 1; layers <= 8; ++layers) {
    expect(true, layers, 12, 12, 13, "a few CTAs");
    expect(true, layers, 400, 400, 13, "one round");
    expect(layers > 4, layers, 2368, 25600, 14, "many rounds");
    expect(layers > 4, layers, 592, 1184, 14, "two even rounds");
    expect(false, layers, 592, 1000, 14, "two uneven rounds");
    expect(false, layers, 592, 592, 22, "long columns");
  }
  if (!failures) std::printf("all ok\n");
  return failures != 0;
}
