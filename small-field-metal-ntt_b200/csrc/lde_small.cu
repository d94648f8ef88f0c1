// lde_small.cu -- coset LDE / blow-up of short columns (2^5 .. 2^14 points) in
// one launch.
//
// A tile is whole columns in one CTA: 2^11 words (2^12 points and up: one
// column), 16 points per thread.  The inverse layers, then per output block q the
// multiplier M_q (BabyBear / KoalaBear) or n^-1 (M31) and the forward layers run
// on the tile engine's rounds (TPass with its own tile size), exchanging
// through shared memory; the inverse result stays in registers across the
// blocks.  The inverse starts and the forward ends in round 0's layout, where a
// thread owns 16 consecutive words, so the input comes straight into registers
// and the output leaves straight from them with 128-bit accesses: no staging
// tile, no tensor maps, no waits on copies.
//
// Small batches are latency: 2^11 x 200, 4x filled 50 CTAs with 2^13-word
// tiles, each running 55 layers in turn and reading one twiddle per butterfly
// from L2 with spilled registers.  Here one column is one CTA, its twiddles
// arrive by asynchronous copies (M31: 128-bit pairs through L1), and while the
// GPU has room the output blocks of a column go to separate CTAs, each repeating
// the inverse (1 + 1 instead of 1 + 2^b transforms in a row).  Device time, before
// -> now, BabyBear: 2^11 x 200 4x 54 -> 9.5 us, 2^12 x 500 8x 223 -> 61 us (28 us
// of butterflies at the integer ceiling, 11 us of output), 2^10 x 1 2x 8.3 -> 2.9
// us, 2^6 x 2001 4x 15.8 -> 4.1 us; M31 / circle, which took three launches:
// 2^11 x 200 4x 23 -> 10 us, 2^12 x 1 2x 13.3 -> 5.8 us, 2^12 x 500 8x 80 -> 66 us.
#include <algorithm>
#include <string>

#include "context.hpp"
#include "pdl.cuh"
#include "tma_launch.cuh"

namespace sfntt {
namespace {

struct SmallLdeArgs {
  const uint32_t* in;
  uint32_t* out;
  uint64_t in_stride;  // column stride in words, a multiple of 4
  const uint2* tw_inv;
  const uint2* tw_fwd;
  const uint2* mul;    // BabyBear / KoalaBear: M_q[i] at q n + i
  uint32_t scale_w, scale_ws;  // M31: n^-1
  uint32_t batch, tiles, log_q;
};

// Asynchronous copy of `entries` twiddle pairs (both arrays 16-byte aligned)
// into shared memory, committed as one group per thread: every load is in
// flight at once and the wait sits where the first twiddle is needed.
template <uint32_t ENTRIES, uint32_t NT>
__device__ __forceinline__ void stage_async(uint2* dst, const uint2* src, uint32_t tid) {
  const uint32_t d = tma::smem_addr(dst);
#pragma unroll
  for (uint32_t i = 0; i < (ENTRIES / 2 + NT - 1) / NT; ++i) {
    const uint32_t v = tid + i * NT;
    if (v < ENTRIES / 2)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16u * v), "l"(src + 2u * v) : "memory");
  }
  if ((ENTRIES & 1u) && tid == 0)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d + 8u * (ENTRIES - 1u)), "l"(src + ENTRIES - 1u)
                 : "memory");
  asm volatile("cp.async.commit_group;" ::: "memory");
}

constexpr int small_tile_bits(int P) { return P > 11 ? P : 11; }

template <class F, int P>
struct SmallLde {
  static constexpr int TB = small_tile_bits(P);
  using Inv = TPass<F, false, Kind::C, P, false, false, false, false, TB>;
  using Fwd = TPass<F, true, Kind::C, P, false, false, false, false, TB>;
  static constexpr int K = Inv::K, E = Inv::E, NT = Inv::NT;
  static constexpr uint32_t N = 1u << P;
  static constexpr int kCtasPerSm = NT <= 128 ? 4 : NT <= 256 ? 2 : 1;  // registers: 128 per thread (1024 threads: 64)
  static constexpr uint32_t TW_ENTRIES = Inv::TW_ENTRIES;  // per direction (M31: none)
  static constexpr uint32_t TW_STRIDE = (TW_ENTRIES + 1u) & ~1u;  // 16-byte aligned tables
  static constexpr int kSmemBytes = (int)(4u * Inv::TWORDS + 16u * TW_STRIDE);
  static_assert(RM<Kind::C, P, TB - P, 4, 0>::cm(15) == 15u, "round 0: 16 consecutive words per thread");
  static_assert(Inv::kFirst == 0 && Fwd::kLast == 0, "round 0 at both ends");
  using M = RM<Kind::C, P, TB - P, 4, K - 1>;
  // the next block's multipliers wait in registers while a block's layers run,
  // where the CTA's registers allow (1024 threads: 64 each)
  static constexpr bool kPrefetch = F::kMontgomery && NT <= 512;

  // Where the multiplier of column position i sits in block q's table: position
  // order (kind 0) up to 2^13 points, the TMA expansion's tile order (kind 2; at
  // 2^13 points the same) from there on, so both routes of a size read one table.
  __device__ static constexpr uint32_t mul_at(uint32_t i) {
    return P == 14 ? ((i & 31u) | ((i >> 6) << 5) | (((i >> 5) & 1u) << 13)) : i;
  }
  __device__ static __forceinline__ void load_mul(uint2 (&w)[E], const uint2* mq) {
#pragma unroll
    for (int m = 0; m < E; ++m) w[m] = __ldg(mq + mul_at(M::cm(m) & (N - 1u)));
  }

  __device__ static void run(const SmallLdeArgs& a) {
    extern __shared__ __align__(1024) uint32_t smem_words[];
    uint32_t* buf = smem_words;
    uint2* tws_inv = reinterpret_cast<uint2*>(buf + Inv::TWORDS);
    uint2* tws_fwd = tws_inv + TW_STRIDE;
    const uint32_t tid = threadIdx.x;
    if constexpr (Inv::kStaged) {
      stage_async<TW_ENTRIES, NT>(tws_inv, a.tw_inv, tid);
      stage_async<TW_ENTRIES, NT>(tws_fwd, a.tw_fwd, tid);
    }
    bool first = true;
    TmaArgs ai{}, af{};
    ai.tw = a.tw_inv;
    ai.log_n = P;
    af.tw = a.tw_fwd;
    af.log_n = P + a.log_q;
    const uint32_t nq = 1u << a.log_q;
    const uint32_t c0 = 16u * tid;                     // the thread's words in round 0's layout
    const uint32_t ct = mul_at(M::ctid(tid) & (N - 1u));  // multiplier of its slot 0 in round K-1's
    const TileCoord gi{};
    for (uint32_t t = blockIdx.x; t < a.tiles; t += gridDim.x) {
      const uint32_t col = (t << (TB - P)) + (c0 >> P);
      const uint32_t row = c0 & (N - 1u);
      const bool live = col < a.batch;  // the last tile may hold fewer columns
      uint32_t x[E], v[E];
      const uint4* src = reinterpret_cast<const uint4*>(a.in + (uint64_t)col * a.in_stride + row);
#pragma unroll
      for (int m = 0; m < E; m += 4) {
        const uint4 q = live ? src[m >> 2] : make_uint4(0, 0, 0, 0);
        x[m] = q.x; x[m + 1] = q.y; x[m + 2] = q.z; x[m + 3] = q.w;
      }
      uint2 w[kPrefetch ? E : 1];
      if constexpr (kPrefetch) load_mul(w, a.mul + (uint64_t)blockIdx.y * N + ct);  // in flight during the inverse
      if (Inv::kStaged && first) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");  // the inverse layers' twiddles
        __syncthreads();
      }
      Inv::template rounds<0>(buf, x, ai, tws_inv, gi, tid);  // x: round K-1 layout
      if constexpr (!F::kMontgomery) {
#pragma unroll
        for (int m = 0; m < E; ++m) x[m] = mul_shoup<F>(x[m], a.scale_w, a.scale_ws);
      }
      if (Inv::kStaged && first) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");  // the forward layers' twiddles
        __syncthreads();
      }
      first = false;
      for (uint32_t q = blockIdx.y; q < nq; q += gridDim.y) {
        if constexpr (F::kMontgomery && !kPrefetch) {
          const uint2* mq = a.mul + (uint64_t)q * N + ct;
#pragma unroll
          for (int m = 0; m < E; ++m) {
            const uint2 wm = __ldg(mq + mul_at(M::cm(m) & (N - 1u)));
            v[m] = mul_shoup<F>(x[m], wm.x, wm.y);
          }
        } else if constexpr (F::kMontgomery) {
#pragma unroll
          for (int m = 0; m < E; ++m) v[m] = mul_shoup<F>(x[m], w[m].x, w[m].y);
          if (q + gridDim.y < nq) load_mul(w, a.mul + (uint64_t)(q + gridDim.y) * N + ct);
        } else {
#pragma unroll
          for (int m = 0; m < E; ++m) v[m] = x[m];
        }
        TileCoord gq{};
        gq.pos_base = q << P;  // M31: block q of the extended network
        Fwd::template rounds<0>(buf, v, af, tws_fwd, gq, tid);  // ends in round 0's layout
        if constexpr (!Net<F, true>::kGS) {
#pragma unroll
          for (int m = 0; m < E; ++m) v[m] = reduce2p<F>(v[m]);
        }
        if (live) {
          uint4* dst = reinterpret_cast<uint4*>(a.out + (((uint64_t)col << a.log_q) + q) * N + row);
#pragma unroll
          for (int m = 0; m < E; m += 4) dst[m >> 2] = make_uint4(v[m], v[m + 1], v[m + 2], v[m + 3]);
        }
        // The next block (or tile) writes words in round K-1's (0's) layout that
        // other threads may still be reading in this block's last round.
        __syncthreads();
      }
    }
  }
};

template <class F, int P>
__global__ void __launch_bounds__(SmallLde<F, P>::NT, SmallLde<F, P>::kCtasPerSm) lde_small_kernel(SmallLdeArgs a) {
  pdl_enter();
  SmallLde<F, P>::run(a);
}

template <class F, int P>
Status launch(sfntt_ctx* ctx, SmallLdeArgs a, bool split, cudaStream_t s) {
  using L = SmallLde<F, P>;
  a.tiles = (uint32_t)((((uint64_t)a.batch << P) + L::Inv::TWORDS - 1) >> L::TB);
  auto kern = lde_small_kernel<F, P>;
  static std::atomic<uint64_t> smem_done{0};
  SFNTT_TRY(smem_limit_once(kern, L::kSmemBytes, ctx->device, smem_done));
  // CTAs per SM: shared memory (1 KiB reserved each) and the launch bounds' registers
  const uint32_t per_sm = std::min<uint32_t>(L::kCtasPerSm, 233472u / (uint32_t)(L::kSmemBytes + 1024));
  const uint32_t room = per_sm * (uint32_t)ctx->sm_count;
  dim3 grid(std::min<uint32_t>(a.tiles, room));
  // Output blocks of a column on separate CTAs, each repeating the inverse, in the
  // split that takes the fewest transforms in a row: while every CTA has a place
  // that costs nothing, and past that it evens out a last round of few tiles (M31
  // 2^13 x 150 16x, one CTA per SM: two rounds of 17 transforms 147 us, five of 5
  // 110 us; 2^12 x 150 16x, two per SM: 62 -> 45 us).  Several rounds of two or more
  // CTAs per SM fill in by themselves (2^12 x 400 4x 29.5 against 33 us split).  Not
  // when the input lies in the output columns, which another CTA would overwrite.
  if (split) {
    const uint32_t nq = 1u << a.log_q;
    const bool uneven = per_sm == 1 || a.tiles <= room;
    uint64_t best = 0;
    for (uint32_t y = 1; y <= nq; y *= 2) {
      const uint64_t rounds = ((uint64_t)a.tiles * y + room - 1) / room;
      const uint64_t row = rounds * (1u + nq / y);
      if (y == 1 || (rounds == 1 && row < best) || (uneven && 20 * row < 19 * best)) {
        best = row;
        grid.x = y == 1 ? std::min<uint32_t>(a.tiles, room) : a.tiles;
        grid.y = y;
      }
    }
  }
  launch_begin(ctx, s);
  SFNTT_CU(launch_pdl(kern, grid, L::NT, L::kSmemBytes, s, (uint64_t)grid.x * grid.y <= 16, a));
  static const std::string name = std::string(F::kTag) + "_lde_small_C" + std::to_string(P);
  return launch_check(ctx, name.c_str(), s, ((uint64_t)a.batch << P) * 4u * (1u + (1u << a.log_q)));
}

template <class F>
Status dispatch(sfntt_ctx* ctx, uint32_t log_n, const SmallLdeArgs& a, bool split, cudaStream_t s) {
  switch (log_n) {
    case 5: return launch<F, 5>(ctx, a, split, s);
    case 6: return launch<F, 6>(ctx, a, split, s);
    case 7: return launch<F, 7>(ctx, a, split, s);
    case 8: return launch<F, 8>(ctx, a, split, s);
    case 9: return launch<F, 9>(ctx, a, split, s);
    case 10: return launch<F, 10>(ctx, a, split, s);
    case 11: return launch<F, 11>(ctx, a, split, s);
    case 12: return launch<F, 12>(ctx, a, split, s);
    case 13: return launch<F, 13>(ctx, a, split, s);
    case 14: return launch<F, 14>(ctx, a, split, s);
    default: return {SFNTT_INVALID_ARGUMENT, "short-column LDE: 2^5 .. 2^14 points"};
  }
}

}  // namespace

// 2^13 points replace three launches by one at every batch (BabyBear 2x: 1
// column 16.5 -> 9.4 us, 40 19.9 -> 10.1 us, 1000 95.9 -> 84.5 us).  2^14 points
// leave one 1024-thread CTA per SM, which only wins while every output block
// has an SM to itself (40 columns 2x 21.5 -> 18.2 us, 10 columns 4x 23.9 ->
// 17.9 us; 150 columns 2x 41.9 -> 49.8 us).
bool lde_small_fits(const sfntt_ctx* ctx, const uint32_t* in, const uint32_t* out, uint64_t in_stride, uint32_t log_n,
                    uint32_t batch, uint32_t added_bits) {
  if (ctx->no_tma || log_n < 5 || log_n > 14 || added_bits > 4) return false;
  if (!aligned16(in) || !aligned16(out) || (in_stride & 3u) != 0) return false;
  // Nothing orders one CTA's reads against another's stores: an input that lies
  // in the output must be read and overwritten by the same CTA, column by column
  // (the natural-order route, or one column); the passes take any other overlap.
  const uintptr_t ib = reinterpret_cast<uintptr_t>(in), ob = reinterpret_cast<uintptr_t>(out);
  const uint64_t n = 1ull << log_n, n_ext = n << added_bits;
  const uint64_t in_bytes = 4 * ((batch - 1ull) * in_stride + n), out_bytes = 4 * batch * n_ext;
  if (ib < ob + out_bytes && ob < ib + in_bytes && !(ib == ob && (batch == 1 || in_stride == n_ext))) return false;
  return log_n < 14 || (in != out && ((uint64_t)batch << added_bits) <= (uint64_t)ctx->sm_count);
}

Status lde_small_dev(sfntt_ctx* ctx, int field, const uint32_t* in, uint64_t in_stride, uint32_t* out, uint32_t log_n,
                     uint32_t batch, uint32_t added_bits, const uint2* tw_inv, const uint2* tw_fwd, const uint2* mul,
                     uint32_t scale_w, cudaStream_t s) {
  SmallLdeArgs a{};
  a.in = in;
  a.out = out;
  a.in_stride = in_stride;
  a.tw_inv = tw_inv;
  a.tw_fwd = tw_fwd;
  a.mul = mul;
  a.scale_w = scale_w;
  a.batch = batch;
  a.log_q = added_bits;
  const bool split = in != out;
  return with_field(field, [&](auto fld) -> Status {
    using F = decltype(fld);
    a.scale_ws = (uint32_t)(((uint64_t)scale_w << 32) / F::P);
    return dispatch<F>(ctx, log_n, a, split, s);
  });
}

}  // namespace sfntt
