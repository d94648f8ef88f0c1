// tma_launch.cuh -- host side of the persistent TMA tile engine: tensor-map
// encoding, shape checks and dispatch to the template instantiations.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>

#include <string>

#include "context.hpp"
#include "tile_tma.cuh"
#include "tile_warp.cuh"

namespace sfntt {

struct TmaRequest {
  const uint32_t* in;
  uint32_t* out;
  uint64_t in_stride, out_stride;  // column strides in words
  const uint2* tw;
  uint32_t log_n, lo;
  int P;
  bool contiguous;
  uint32_t batch;
  uint32_t scale_w;  // canonical multiplier for the outputs; 0 = none
  const uint2* twist = nullptr;  // BabyBear four-step twist at the boundary
  uint32_t twist_mask = 0;
  bool twist_compact = false;    // the twist table holds Shoup companions only (TmaArgs::twist_compact)
  bool plain = false;            // BabyBear strided pass: plain sub-transform (twist by neighbours)
  // per-position twiddles staged in shared memory, one CTA per SM walking the
  // columns (BabyBear 8-layer strided or M31 contiguous passes, n >= 2^13)
  bool lstage = false;
  // M31 over columns of interleaved pairs (CM31): log_n, lo and P count pairs,
  // the strides words
  bool pair = false;
};

// Resolved once through the runtime (no link-time dependency on libcuda).
// swizzle128: 128-byte swizzle of the box in shared memory (16-byte chunk j of
// 128-byte row r lands at chunk j ^ (r & 7); the buffer is 1024-byte aligned).
Status tensor_map_encode(CUtensorMap* map, const void* base, uint32_t rank, const cuuint64_t* dims,
                         const cuuint64_t* strides_bytes, const cuuint32_t* box, bool swizzle128 = false);

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Can a pass of this shape run on the TMA engine?  Contiguous passes over
// columns shorter than a tile need dense columns (stride n) of whole 128-byte
// rows.  A batch that does not fill its last tile takes the engine from 2^18
// words on (n = 2^12: from one tile): the copies fill and clip what lies past
// the end.  Below that the one-group-per-CTA passes of the first engine are
// quicker (BabyBear 2^9 x 41 forward 3.7 against 4.2 us, x 333 4.0 against 4.8
// us; but x 20001 49.0 against 21.3 us, 2^8 x 4001 9.1 against 4.5 us, 2^12 x 3
// 7.6 against 5.9 us).
inline bool tma_pass_ok(const TmaRequest& r) {
  if (!aligned16(r.in) || !aligned16(r.out) || (r.in_stride & 3) || (r.out_stride & 3)) return false;
  const uint32_t pair = r.pair ? 1u : 0u;
  const uint64_t n = 1ull << (r.log_n + pair);  // words per column
  if (r.contiguous) {
    if (r.P < 5 || r.P > (r.pair ? 12 : 14) || r.lo != 0) return false;
    if (n >= kTileWords) return true;
    const uint64_t words = (uint64_t)r.batch * n;
    return n >= 32 && r.in_stride == n && r.out_stride == n &&
           (words % kTileWords == 0 || words >= (r.log_n + pair >= 12 ? (uint64_t)kTileWords : 1ull << 18));
  }
  return r.P >= 1 && r.P <= 8 && r.lo + pair >= 5 && r.lo + r.P <= r.log_n;
}

// Contiguous tiles of a P-layer pass.  Row order (c_row_perm(P) false):
// box_rows 128-byte rows per copy (a whole 2^13-word tile, or half of one for
// passes that run independent halves).  Row-permuted: a half tile per copy,
// its rows in the order [r0 r1][r3 ..][r2] of the row index r (dims: 32
// words, rows r0..r1, rows r3 and up, row r2, column), whatever box_rows says.
inline Status encode_c_map(CUtensorMap* m, const uint32_t* base, uint32_t log_n, uint64_t stride, uint32_t batch,
                           int P, uint32_t box_rows = kTileWords / 32) {
  const uint64_t n = 1ull << log_n;
  // rows per column and the column stride (dense columns shorter than a tile
  // are one long column)
  const uint64_t rows = n >= kTileWords ? n / 32 : (uint64_t)batch * n / 32;
  const uint64_t cols = n >= kTileWords ? batch : 1;
  const uint64_t col_bytes = n >= kTileWords ? stride * 4 : (uint64_t)batch * n * 4;
  if (c_row_perm(P)) {
    // half a tile per copy: 2^(tile bits - 1) words; 14-layer passes have 2^14-word tiles
    const uint32_t half_words = (P > (int)kTileBits ? (1u << P) : kTileWords) / 2;
    const cuuint64_t dims[5] = {32, 4, rows / 8, 2, cols};
    const cuuint64_t strides[4] = {128, 1024, 512, col_bytes};
    const cuuint32_t box[5] = {32, 4, half_words / 256, 2, 1};
    return tensor_map_encode(m, base, 5, dims, strides, box, kSwizzleC);
  }
  const cuuint64_t dims[3] = {32, rows, cols};
  const cuuint64_t strides[2] = {128, col_bytes};
  const cuuint32_t box[3] = {32, box_rows, 1};
  return tensor_map_encode(m, base, 3, dims, strides, box, kSwizzleC);
}

// column viewed as [hb][e][lchunk][u]: u 32 words, lchunk 2^lo/32, e 2^P (stride 2^lo), hb
inline Status encode_s_map(CUtensorMap* m, const uint32_t* base, uint32_t lo, int P, uint64_t hb_count,
                           uint64_t hb_stride, uint64_t stride, uint32_t batch) {
  const cuuint64_t dims[5] = {32, (1ull << lo) / 32, 1ull << P, hb_count, batch};
  const cuuint64_t strides[4] = {128, (1ull << lo) * 4, hb_stride * 4, stride * 4};
  const cuuint32_t box[5] = {32, 1, (cuuint32_t)(1u << P), 1, 1};
  return tensor_map_encode(m, base, 5, dims, strides, box);
}

// The same strided tiles of 8 layers for the warp-owned passes: positions as one
// dimension, the element in two, in the row order of tile_warp.cuh.
inline Status encode_w_map(CUtensorMap* m, const uint32_t* base, uint32_t lo, wt::RowOrder order, uint64_t hb_count,
                           uint64_t hb_stride, uint64_t stride, uint32_t batch) {
  const cuuint64_t elo = (4ull << lo), ehi = (64ull << lo);  // byte strides of e + 1, e + 16
  const cuuint64_t dims[5] = {1ull << lo, 16, 16, hb_count, batch};
  const cuuint64_t strides[4] = {order == wt::kSwapped ? ehi : elo, order == wt::kSwapped ? elo : ehi, hb_stride * 4,
                                 stride * 4};
  const cuuint32_t box[5] = {32, 16, 16, 1, 1};
  return tensor_map_encode(m, base, 5, dims, strides, box, true);
}

// The passes that take the warp-owned tiles: the network's top 8 layers without
// a boundary twist, at least three tiles per SM (see tile_warp.cuh).
template <class F>
bool warp_pass_ok(const sfntt_ctx* ctx, const TmaRequest& r) {
  return (F::kMontgomery ? r.plain && !r.twist : !r.twist) && r.lo + 8 == r.log_n &&
         (((uint64_t)r.batch << (r.log_n + (r.pair ? 1 : 0))) >> kTileBits) >= 3ull * (uint64_t)ctx->sm_count;
}

template <class F, bool DESC>
Status launch_warp_pass(sfntt_ctx* ctx, const TmaRequest& r, cudaStream_t s) {
  using W = WPass<F, DESC>;
  const uint32_t pair = r.pair ? 1u : 0u, log_w = r.log_n + pair, lo_w = r.lo + pair;
  CUtensorMap min, mout;
  SFNTT_TRY(encode_w_map(&min, r.in, lo_w, W::kIn, 1, 1ull << log_w, r.in_stride, r.batch));
  SFNTT_TRY(encode_w_map(&mout, r.out, lo_w, W::kOut, 1, 1ull << log_w, r.out_stride, r.batch));
  TmaArgs a{};
  a.tw = r.tw;
  a.log_n = r.log_n;
  a.lo = r.lo;
  a.pair = pair;
  a.batch = r.batch;
  a.err = ctx->err.as<int>();
  a.scale = r.scale_w ? 1u : 0u;
  a.scale_w = r.scale_w;
  a.scale_ws = (uint32_t)(((uint64_t)r.scale_w << 32) / F::P);
  a.ntiles = (uint32_t)(((uint64_t)r.batch << log_w) >> kTileBits);
  auto kern = warp_pass_kernel<F, DESC>;
  static std::atomic<uint64_t> smem_done{0};
  SFNTT_TRY(smem_limit_once(kern, W::kSmemBytes, ctx->device, smem_done));
  const uint32_t ctas = ctx->tma_ctas > 0 ? std::min<uint32_t>((uint32_t)ctx->tma_ctas, wt::kCtasPerSm) : wt::kCtasPerSm;
  const uint32_t grid = std::min<uint32_t>(a.ntiles, ctas * (uint32_t)ctx->sm_count);
  launch_begin(ctx, s);
  SFNTT_CU(launch_pdl(kern, grid, wt::kThreads, W::kSmemBytes, s, pdl_fits(grid, a.ntiles, a.log_n), min, mout, a));
  static const std::string name = std::string(F::kTag) + (DESC ? "_fwd" : "_inv") + "_warp_S8" + (F::kMontgomery ? "p" : "");
  return launch_check(ctx, name.c_str(), s, ((uint64_t)r.batch << log_w) * 8u);
}

template <class F, bool DESC, Kind KD, int P, bool PLAIN, bool TW, bool LSTAGE>
const char* tma_pass_name() {
  static const std::string nm = std::string(F::kTag) + "_" + (DESC ? "fwd" : "inv") +
                                "_tma_" + (KD == Kind::C ? "C" : KD == Kind::D ? "D" : "S") + std::to_string(P) + (PLAIN ? "p" : "") +
                                (TW ? "t" : "") + (LSTAGE ? "c" : "");
  return nm.c_str();
}

template <class F, bool DESC, Kind KD, int P, bool PLAIN, bool TW, bool LSTAGE = false, bool HALVES = false>
Status launch_tma_pass(sfntt_ctx* ctx, const TmaRequest& r, cudaStream_t s) {
  using T = TPass<F, DESC, KD, P, PLAIN, TW, LSTAGE, HALVES>;
  const uint32_t pair = r.pair ? 1u : 0u;
  const uint32_t log_w = r.log_n + pair, lo_w = r.lo + pair;  // in words
  const uint64_t n = 1ull << log_w;
  CUtensorMap min, mout;
  TmaArgs a{};
  a.pair = pair;
  a.tw = r.tw;
  a.log_n = r.log_n;
  a.lo = r.lo;
  a.batch = r.batch;
  a.err = ctx->err.as<int>();
  a.scale = r.scale_w ? 1u : 0u;
  a.scale_w = r.scale_w;
  a.scale_ws = (uint32_t)(((uint64_t)r.scale_w << 32) / F::P);
  a.twist = r.twist;
  a.twist_mask = r.twist_mask;
  a.twist_compact = r.twist_compact ? 1u : 0u;
  if constexpr (KD != Kind::S) {
    const uint32_t rows = HALVES ? T::HROWS : T::TWORDS / 32;
    const int order = KD == Kind::C ? P : 0;  // rows of pair tiles stay in order
    SFNTT_TRY(encode_c_map(&min, r.in, log_w, r.in_stride, r.batch, order, rows));
    SFNTT_TRY(encode_c_map(&mout, r.out, log_w, r.out_stride, r.batch, order, rows));
    a.spans = n < T::TWORDS;
    a.log_tpc = a.spans ? 0u : log_w - T::CB;
    // every M31 table with n >= 2^13 carries its first-round copy from entry n on
    if constexpr (T::kRound0Copy) a.tw0 = a.spans ? nullptr : r.tw + n;
    a.ntiles = (uint32_t)(((uint64_t)r.batch * n + T::TWORDS - 1) >> T::CB);
  } else {
    const uint64_t hb = n >> (lo_w + P);
    SFNTT_TRY(encode_s_map(&min, r.in, lo_w, P, hb, 1ull << (lo_w + P), r.in_stride, r.batch));
    SFNTT_TRY(encode_s_map(&mout, r.out, lo_w, P, hb, 1ull << (lo_w + P), r.out_stride, r.batch));
    a.ntiles = (uint32_t)(((uint64_t)r.batch * n) >> (P + 5));
  }
  constexpr int smem = T::kSmemBytes;
  auto kern = tma_pass_kernel<F, DESC, KD, P, PLAIN, TW, LSTAGE, HALVES>;
  static std::atomic<uint64_t> smem_done{0};
  SFNTT_TRY(smem_limit_once(kern, smem, ctx->device, smem_done));
  const uint32_t ctas = ctx->tma_ctas > 0 ? std::min<uint32_t>((uint32_t)ctx->tma_ctas, T::kCtasPerSm) : T::kCtasPerSm;
  const uint32_t grid = std::min<uint32_t>(a.ntiles, ctas * (uint32_t)ctx->sm_count);
  launch_begin(ctx, s);
  // (LSTAGE: contiguous ranges of tiles per CTA, where an early launch gained nothing)
  const bool early = LSTAGE ? grid <= 16 : KD == Kind::S ? pdl_fits_strided(P, grid, a.ntiles, a.log_n) : pdl_fits(grid, a.ntiles, a.log_n);
  SFNTT_CU(launch_pdl(kern, grid, T::NT, smem, s, early, min, mout, a));
  return launch_check(ctx, tma_pass_name<F, DESC, KD, P, PLAIN, TW, LSTAGE>(), s,
                      ((uint64_t)r.batch << log_w) * 8u);
}

// BabyBear and KoalaBear instantiate the twist / plain variants; M31 never needs them.
#define SFNTT_TMA_C(PP)                                                                          \
  case PP:                                                                                       \
    if constexpr (F::kMontgomery) {                                                              \
      if (r.twist) {                                                                             \
        if constexpr (TPass<F, DESC, Kind::C, PP, false, true>::halves_ok())                     \
          if (ctx->c_halves) return launch_tma_pass<F, DESC, Kind::C, PP, false, true, false, true>(ctx, r, s); \
        return launch_tma_pass<F, DESC, Kind::C, PP, false, true>(ctx, r, s);                    \
      }                                                                                          \
    } else {                                                                                     \
      if (r.lstage && r.log_n >= kTileBits)                                                      \
        return launch_tma_pass<F, DESC, Kind::C, PP, false, false, true>(ctx, r, s);             \
    }                                                                                            \
    if constexpr (TPass<F, DESC, Kind::C, PP, false, false>::halves_ok())                        \
      if (ctx->c_halves) return launch_tma_pass<F, DESC, Kind::C, PP, false, false, false, true>(ctx, r, s); \
    return launch_tma_pass<F, DESC, Kind::C, PP, false, false>(ctx, r, s);
#define SFNTT_TMA_S(PP)                                                                          \
  case PP:                                                                                       \
    if constexpr (PP == 8) {                                                                     \
      if (warp_pass_ok<F>(ctx, r)) return launch_warp_pass<F, DESC>(ctx, r, s);                  \
    }                                                                                            \
    if constexpr (F::kMontgomery) {                                                              \
      if (r.plain && r.twist) return launch_tma_pass<F, DESC, Kind::S, PP, true, true>(ctx, r, s); \
      if (r.plain) return launch_tma_pass<F, DESC, Kind::S, PP, true, false>(ctx, r, s);         \
      if (r.twist) return launch_tma_pass<F, DESC, Kind::S, PP, false, true>(ctx, r, s);         \
      if constexpr (PP == 8) {                                                                   \
        if (r.lstage) return launch_tma_pass<F, DESC, Kind::S, PP, false, false, true>(ctx, r, s); \
      }                                                                                          \
    }                                                                                            \
    return launch_tma_pass<F, DESC, Kind::S, PP, false, false>(ctx, r, s);

#define SFNTT_TMA_D(PP)                                                                          \
  case PP:                                                                                       \
    if (r.lstage && r.log_n + 1 >= kTileBits)                                                    \
      return launch_tma_pass<F, DESC, Kind::D, PP, false, false, true>(ctx, r, s);               \
    return launch_tma_pass<F, DESC, Kind::D, PP, false, false>(ctx, r, s);

template <class F, bool DESC>
Status run_tma_pass_impl(sfntt_ctx* ctx, const TmaRequest& r, cudaStream_t s) {
  if (!tma_pass_ok(r)) return {SFNTT_INVALID_ARGUMENT, "pass shape not supported by the TMA engine"};
  if (r.pair && F::kMontgomery) return {SFNTT_INVALID_ARGUMENT, "passes over pairs are M31"};
  if constexpr (!F::kMontgomery) {
    if (r.pair && r.contiguous) {
      switch (r.P) {
        SFNTT_TMA_D(5) SFNTT_TMA_D(6) SFNTT_TMA_D(7) SFNTT_TMA_D(8)
        SFNTT_TMA_D(9) SFNTT_TMA_D(10) SFNTT_TMA_D(11) SFNTT_TMA_D(12)
        default: break;
      }
    }
  }
  if (!F::kMontgomery && (r.twist || r.plain)) return {SFNTT_INVALID_ARGUMENT, "M31 passes take no twist"};
  if (r.contiguous) {
    switch (r.P) {
      SFNTT_TMA_C(5) SFNTT_TMA_C(6) SFNTT_TMA_C(7) SFNTT_TMA_C(8)
      SFNTT_TMA_C(9) SFNTT_TMA_C(10) SFNTT_TMA_C(11) SFNTT_TMA_C(12) SFNTT_TMA_C(13)
      SFNTT_TMA_C(14)
      default: break;
    }
  } else {
    switch (r.P) {
      SFNTT_TMA_S(1) SFNTT_TMA_S(2) SFNTT_TMA_S(3) SFNTT_TMA_S(4)
      SFNTT_TMA_S(5) SFNTT_TMA_S(6) SFNTT_TMA_S(7) SFNTT_TMA_S(8)
      default: break;
    }
  }
  return {SFNTT_INVALID_ARGUMENT, "unsupported TMA pass size"};
}
#undef SFNTT_TMA_C
#undef SFNTT_TMA_S
#undef SFNTT_TMA_D

Status run_tma_pass_bb_fwd(sfntt_ctx* ctx, const TmaRequest& r, cudaStream_t s);
Status run_tma_pass_bb_inv(sfntt_ctx* ctx, const TmaRequest& r, cudaStream_t s);
Status run_tma_pass_kb_fwd(sfntt_ctx* ctx, const TmaRequest& r, cudaStream_t s);
Status run_tma_pass_kb_inv(sfntt_ctx* ctx, const TmaRequest& r, cudaStream_t s);
Status run_tma_pass_m31_fwd(sfntt_ctx* ctx, const TmaRequest& r, cudaStream_t s);
Status run_tma_pass_m31_inv(sfntt_ctx* ctx, const TmaRequest& r, cudaStream_t s);

inline Status run_tma_pass_field(sfntt_ctx* ctx, int field, bool desc, const TmaRequest& r, cudaStream_t s) {
  if (field == SFNTT_BABYBEAR) return desc ? run_tma_pass_bb_fwd(ctx, r, s) : run_tma_pass_bb_inv(ctx, r, s);
  if (field == SFNTT_KOALABEAR) return desc ? run_tma_pass_kb_fwd(ctx, r, s) : run_tma_pass_kb_inv(ctx, r, s);
  return desc ? run_tma_pass_m31_fwd(ctx, r, s) : run_tma_pass_m31_inv(ctx, r, s);
}

}  // namespace sfntt
