// pdl.cuh -- programmatic dependent launch between consecutive passes.
//
// A pass launched with launch_pdl may be scheduled while the previous kernel
// on its stream is still running: once every CTA of that kernel has issued its
// trigger (or ended), the pass's CTAs take the SM slots that come free, run
// their prologue (barriers, tensor maps, twiddles staged from tables that no
// kernel in flight writes) and wait (griddepcontrol.wait) until every
// prerequisite grid has completed and its writes are visible, before touching
// data.  The launch gap and the prologue then overlap the previous kernel's
// end; the ordering of memory effects is that of a plain stream.  A kernel
// launched without the attribute (or after a non-kernel operation) passes the
// wait at once.
//
// Small kernels trigger at their start; the persistent passes when a CTA starts
// its last tile.  (Triggered at the start, a next grid waiting in every free slot
// slowed the full four-step passes by 10 %.)  A persistent grid launched early
// fills slots in the order they come free, so CTAs with one tile more than others
// can end up on one SM: pdl_fits takes the grids whose tiles divide evenly and
// those of eight rounds or more.  Forward + inverse, plain -> early launch:
// BabyBear 2^20 x 1 24.4 -> 21.4 us, KoalaBear 2^17 x 37 48.0 -> 44.9 us, BabyBear
// 2^19 x 64 281 -> 274 us, M31 blow-up 2^16 x 100 85 -> 82 us; not taken: 2^24 x 1
// (6.9 rounds) 209 -> 213 us, CM31 2^16 x 24 (1.3 rounds) 43 -> 46 us.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <utility>

namespace sfntt {

// First statement of every kernel launched with launch_pdl (or the two halves,
// with loads of tables -- finished before any launch that uses them -- between).
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_enter() {
  pdl_trigger();
  pdl_wait();
}

// PDL for a grid of `ctas` CTAs over `tiles` tiles of columns of 2^log_n words.
// Not from 2^22 words on: there an early launch gains nothing and mostly loses
// (plain -> early: BabyBear LDE 2^22 x 64 3.75 -> 3.93 ms, 2^23 x 4 626 -> 668 us,
// 2^21 x 8, whose output has 2^22, 280 -> 295 us, 2^23 x 9 forward 424 -> 438 us).
inline bool pdl_fits(uint64_t ctas, uint64_t tiles, uint32_t log_n) {
  return log_n < 22 && (ctas <= 16 || tiles % ctas == 0 || tiles >= 8 * ctas);
}

// A strided pass of `layers` layers.  Up to four, a tile takes so little time that
// the CTAs of several rounds, launched early into slots that come free one by one,
// run worse than a grid that starts together: natural-order LDE 2^13 x 100 31.2 ->
// 37.0 us, x 2001 383 -> 526 us, 2^15 x 200 107 -> 122 us, 2^16 x 500 407 -> 420 us;
// grids of one round gain (2^13 x 3 17.3 -> 15.2 us), and from five layers on all
// (2^17 x 100 166 -> 164 us).
inline bool pdl_fits_strided(int layers, uint64_t ctas, uint64_t tiles, uint32_t log_n) {
  return (layers > 4 || tiles <= ctas) && pdl_fits(ctas, tiles, log_n);
}

// An expansion of fewer tiles than `slots` (CTAs that fit the GPU) launched early
// packs onto the SMs that come free first: M31 2^16 x 12 4x 28.6 -> 38.5 us.
inline bool pdl_fits_expand(uint64_t ctas, uint64_t tiles, uint64_t slots, uint32_t log_n) {
  return (ctas <= 16 || ctas == slots) && pdl_fits(ctas, tiles, log_n);
}

template <class... KArgs, class... Args>
inline cudaError_t launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, bool pdl,
                              Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
#ifdef SFNTT_NO_PDL  // plain stream ordering (for comparisons)
  cfg.numAttrs = 0;
#else
  cfg.numAttrs = pdl ? 1 : 0;
#endif
  return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

}  // namespace sfntt
