// tile_warp.cuh -- 8-layer strided passes whose warps never wait for one another.
//
// A strided tile is 32 consecutive positions x 256 group elements e (stride
// 2^lo), as in tile_tma.cuh.  Its positions do not interact, so a warp can own 4
// of them for all 256 elements: 32 lanes x (16 elements x 2 neighbouring
// positions) = 1024 words.  Two rounds of 4 layers run in registers; the
// exchange between them stays inside the warp's own words of the tile
// (__syncwarp, 64-bit accesses).  A ninth warp moves the tiles: it brings them
// in by TMA and stores them back when the eight compute warps have arrived on
// the tile's mbarrier, so no CTA-wide barrier exists and the warps drift apart
// until the integer pipes stay busy.  The whole-CTA exchanges and pre-store
// barriers of the 512-thread form left them idle a third of the time.
//
// Shared-memory words.  A tile row (one e, 128 bytes) sits at row r, its 16-byte
// chunk j at chunk j ^ (r & 7) (the 128-byte TMA swizzle); warp w owns chunk j = w
// of every row.  With g the 4 element bits on the lanes and s the 4 on the slots,
// a 64-bit access is free of bank conflicts when r & 7 follows g:
//   ends of round 0 (s = e0..3, g = e4..7): rows r = 16 e_lo + e_hi (kSwapped),
//   ends of round 1 (s = e4..7, g = e0..3): rows r = e (kPlain),
//   the exchange, written in one and read in the other:
//     r = 16 e_lo + (e_hi ^ (e_lo & 7)), for both.
// The tile's row order is the tensor map's: e is split into two dimensions.
//
// What it measured against the 512-thread form (TPass, TExpand): the M31
// expansion of 2^20 x 32 190 -> 165 us -- integer-multiply pipe 64 -> 73 % busy,
// warp instructions per warp-butterfly 10.8 -> 8.8 (two positions share every
// twiddle load and address), barrier stalls 0.88 -> 0.01 cycles per issue; the
// M31 blow-up 2^20 x 64 4x 1437 -> 1358 us, the circle LDE 2^20 x 61 840 -> 814
// us, M31 2^18 x 100 130 -> 121 us.  Not taken: twisted passes (a warp's twist
// loads then span 16 rows: 2^24 inverse 108 -> 149 us), several high blocks
// (M31 tables to refill per tile), and grids of fewer than three tiles per SM,
// where one tile's latency counts and 16 warps finish it sooner (M31 2^20 x 1
// forward 11.8 against 12.1 us).  A prefetch of the next tile into L2 changed
// nothing.
//
// Twiddles are the same for every position: BabyBear / KoalaBear plain
// sub-transforms, tw[beta][e mod 2^beta] (the four-step twist is applied at a
// boundary), and M31 per-block, tw[L][block].  One round's do not depend on the
// lane (U: 15 pairs, broadcast), the other's on g alone (V: 15 x 16 pairs).
#pragma once
#include <cstdint>

#include "tile_tma.cuh"

namespace sfntt {

namespace wt {

constexpr int kSlots = 16;              // slots per thread (element bits of a round)
constexpr int kWarps = 8;               // compute warps per tile
constexpr int kThreads = 32 * (kWarps + 1);
constexpr int kRing = 3;                // tile buffers
constexpr uint32_t kTabPairs = 16u + 256u;  // U (15 used) and V (15 x 16 used), as pairs
constexpr int kCtasPerSm = 2;

enum RowOrder { kPlain, kSwapped };

// Table slot of layer j's k-th twiddle (2 consecutive slots load as 128 bits):
// M31 has 2^(3-j) per layer, BabyBear / KoalaBear 2^j.
template <class F>
__host__ __device__ constexpr uint32_t tab_at(int j, int k) {
  return F::kMontgomery ? (uint32_t)((1 << j) + k) : (uint32_t)(16 - (16 >> j) + k);
}
template <class F>
__host__ __device__ constexpr int tab_count(int j) { return F::kMontgomery ? 1 << j : 8 >> j; }
// The round whose twiddles depend on the lane.
template <class F>
__host__ __device__ constexpr int lane_round() { return F::kMontgomery ? 1 : 0; }

// Word address of pair i (a table slot) of lane element g in V.
__device__ __forceinline__ uint32_t v_at(uint32_t i, uint32_t g) { return 16u + (((i >> 1) * 16u + g) << 1) + (i & 1u); }

// Fills one table (U and V) from the layer table `tw`, by `nt` threads; hb: the
// high block (M31).
template <class F>
__device__ __forceinline__ void fill_table(uint2* tab, const uint2* tw, uint32_t log_n, uint32_t lo, uint32_t hb,
                                           uint32_t tid, uint32_t nt) {
  const uint32_t n = 1u << log_n;
  for (uint32_t x = tid; x < 255u; x += nt) {
    if constexpr (F::kMontgomery) {
      const uint32_t beta = 31u - __clz(x + 1u), idx = x + 1u - (1u << beta);  // tw[beta][idx], idx < 2^beta
      const uint2 w = __ldg(tw + x);
      if (beta < 4u) tab[(1u << beta) + idx] = w;
      else tab[v_at((1u << (beta - 4u)) + (idx >> 4), idx & 15u)] = w;
    } else {
      const uint32_t beta = 7u - (31u - __clz(255u - x)), b = x - (256u - (256u >> beta));  // block b < 2^(7 - beta)
      const uint32_t L = lo + beta;
      const uint2 w = __ldg(tw + (n - (n >> L)) + (hb << (7u - beta)) + b);
      if (beta >= 4u) tab[16u - (16u >> (beta - 4u)) + b] = w;
      else tab[v_at(16u - (16u >> beta) + (b & ((8u >> beta) - 1u)), b >> (3u - beta))] = w;
    }
  }
}

// Loads twiddles k = AT .. of layer j into t (all of them): U or V.
template <class F, bool LANE, int j>
__device__ __forceinline__ void load_layer(uint2 (&t)[8], const uint2* tab, uint32_t g) {
  constexpr int cnt = tab_count<F>(j);
#pragma unroll
  for (int k = 0; k < cnt; k += 2) {
    const uint32_t i = tab_at<F>(j, k);
    const uint2* p = LANE ? tab + 16u + (((i >> 1) * 16u + g) << 1) + (i & 1u) : tab + i;
    if constexpr (cnt == 1) {
      t[0] = *p;
    } else {
      const uint4 q = *reinterpret_cast<const uint4*>(p);
      t[k] = make_uint2(q.x, q.y);
      t[k + 1] = make_uint2(q.z, q.w);
    }
  }
}

template <class F, bool DESC, int ROUND, int j>
__device__ __forceinline__ void layer(uint32_t (&v)[32], const uint2* tab, uint32_t g) {
  constexpr bool LANE = ROUND == lane_round<F>();
  uint2 t[8];
  load_layer<F, LANE, j>(t, tab, g);
#pragma unroll
  for (int m = 0; m < kSlots; ++m) {
    if (m & (1 << j)) continue;
    const int k = F::kMontgomery ? (m & ((1 << j) - 1)) : (m >> (j + 1));
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      uint32_t &a = v[2 * m + p], &b = v[2 * (m | (1 << j)) + p];
      if (F::kMontgomery && !LANE && k == 0) butterfly_unit<F, DESC>(a, b);  // tw[beta][0] = 1
      else butterfly<F, DESC>(a, b, t[k]);
    }
  }
}

// The 4 layers of round ROUND (0: element bits 0..3, 1: bits 4..7).
template <class F, bool DESC, int ROUND>
__device__ __forceinline__ void round(uint32_t (&v)[32], const uint2* tab, uint32_t g) {
  if constexpr (DESC) {
    layer<F, DESC, ROUND, 3>(v, tab, g);
    layer<F, DESC, ROUND, 2>(v, tab, g);
    layer<F, DESC, ROUND, 1>(v, tab, g);
    layer<F, DESC, ROUND, 0>(v, tab, g);
  } else {
    layer<F, DESC, ROUND, 0>(v, tab, g);
    layer<F, DESC, ROUND, 1>(v, tab, g);
    layer<F, DESC, ROUND, 2>(v, tab, g);
    layer<F, DESC, ROUND, 3>(v, tab, g);
  }
}

// Where a thread's words sit in a tile buffer (word offsets).
struct Lane {
  uint32_t g;     // element bits on the lanes
  uint32_t io;    // slot 0 at either end of a pass: row g of its order
  uint32_t x0;    // slot 0 of the exchange in round 0's layout (rows 16 s + (g ^ (s & 7)))
  uint32_t x1;    // ... in round 1's (rows 16 g + (s ^ (g & 7)))
  uint32_t pos;   // first of the thread's two positions within the 32
  __device__ __forceinline__ Lane(uint32_t warp, uint32_t lane) {
    const uint32_t h = lane & 1u;
    g = lane >> 1;
    pos = 4u * warp + 2u * h;
    io = g * 32u + ((warp ^ (g & 7u)) << 2) + 2u * h;
    x0 = io;
    x1 = g * 512u + (g & 7u) * 32u + ((warp ^ (g & 7u)) << 2) + 2u * h;
  }
};

// Tile ends: slot s at rows 16 s + g of the end's row order.
__device__ __forceinline__ void ld_io(const uint32_t* buf, uint32_t (&v)[32], const Lane& l) {
#pragma unroll
  for (int s = 0; s < kSlots; ++s) {
    const uint2 q = *reinterpret_cast<const uint2*>(buf + l.io + 512 * s);
    v[2 * s] = q.x;
    v[2 * s + 1] = q.y;
  }
}
__device__ __forceinline__ void st_io(uint32_t* buf, const uint32_t (&v)[32], const Lane& l) {
#pragma unroll
  for (int s = 0; s < kSlots; ++s)
    *reinterpret_cast<uint2*>(buf + l.io + 512 * s) = make_uint2(v[2 * s], v[2 * s + 1]);
}

// Exchange from round FROM's layout to the other's, inside the warp.  A row's
// low bits and its chunk both carry the exclusive or, 32 + 4 words per step.
template <int R>
__device__ __forceinline__ uint32_t x_at(const Lane& l, int s) {
  const uint32_t f = 36u * (uint32_t)(s & 7);
  return R == 0 ? (l.x0 ^ f) + 512u * (uint32_t)s : (l.x1 ^ f) + 32u * (uint32_t)(s & 8);
}
template <int FROM>
__device__ __forceinline__ void exchange(uint32_t* buf, uint32_t (&v)[32], const Lane& l) {
  __syncwarp();  // every lane has read the words that are overwritten now
#pragma unroll
  for (int s = 0; s < kSlots; ++s)
    *reinterpret_cast<uint2*>(buf + x_at<FROM>(l, s)) = make_uint2(v[2 * s], v[2 * s + 1]);
  __syncwarp();
#pragma unroll
  for (int s = 0; s < kSlots; ++s) {
    const uint2 q = *reinterpret_cast<const uint2*>(buf + x_at<1 - FROM>(l, s));
    v[2 * s] = q.x;
    v[2 * s + 1] = q.y;
  }
  __syncwarp();  // before the words are written again
}

struct Bars {
  uint64_t full[kRing];   // a tile has arrived (transaction bytes)
  uint64_t done[kRing];   // the compute warps have written a block
  uint64_t empty[kRing];  // a block's store has read its buffer
};

__device__ __forceinline__ void init_bars(Bars* b) {
  for (int i = 0; i < kRing; ++i) {
    tma::mbar_init(&b->full[i], 1);
    tma::mbar_init(&b->done[i], kWarps);
    tma::mbar_init(&b->empty[i], 1);
  }
  tma::fence_mbar_init();
}

struct Coord { uint32_t chunk, col; };
// Tile t: column-fastest, then the 32-position chunk (one high block).
__device__ __forceinline__ Coord coord(const TmaArgs& a, uint32_t t) {
  const uint32_t chunk = t / a.batch;
  return {chunk, t - chunk * a.batch};
}

// The ninth warp (one thread).  Output blocks, nq per tile, take the ring's
// buffers in order; block 0 of a tile sits in the buffer its tile arrived in.
// Buffer use u of slot i ends when its store has read it: then compute warps
// may write the block 3 later there, or the tile that starts 3 later is loaded.
template <class StoreFn>
__device__ __forceinline__ void producer(const CUtensorMap* min, uint32_t* ring, Bars* b, const TmaArgs& a, uint32_t nq,
                                         StoreFn store) {
  const uint32_t step = gridDim.x;
  if (blockIdx.x >= a.ntiles) return;
  const uint32_t tiles = (a.ntiles - blockIdx.x + step - 1) / step;  // of this CTA
  const uint32_t blocks = tiles * nq;
  auto load = [&](uint32_t it, uint32_t slot) {
    const Coord c = coord(a, blockIdx.x + it * step);
    tma::mbar_expect_tx(&b->full[slot], kTileBytes);
    tma::load_5d(ring + slot * kTileWords, min, (int32_t)(c.chunk << 5), 0, 0, 0, (int32_t)c.col, &b->full[slot]);
  };
  for (uint32_t i = 0; i < (uint32_t)kRing; ++i)
    if (i % nq == 0 && i / nq < tiles) load(i / nq, i);
  uint32_t slot = 0, use = 0;  // of block k
  for (uint32_t k = 0; k < blocks; ++k) {
    if (!tma::mbar_wait(&b->done[slot], use & 1u, kWaitNs)) {
      atomicExch(a.err, 1);
      // the loads in flight: tiles up to the one that block k + 2 belongs to
      for (uint32_t m = k; m < k + kRing && m < blocks; ++m)
        if (m % nq == 0) tma::mbar_wait(&b->full[m % kRing], (m / nq / kRing) & 1u, kWaitNs);
      break;
    }
    store(k / nq, k % nq, ring + slot * kTileWords);
    tma::commit();
    tma::wait_reads();
    tma::mbar_arrive(&b->empty[slot]);
    const uint32_t next = k + kRing;
    if (next < blocks && next % nq == 0) load(next / nq, slot);
    if (++slot == (uint32_t)kRing) { slot = 0; ++use; }
  }
  tma::wait_all();
}

// A compute warp's wait for a phase of `bar`.  false: it ran out for a lane; the
// flag is set and the warp leaves without arriving again, so nothing of that
// block or of later ones is stored, and the mover's next wait for the warps is
// its last: at most one wait per thread runs out.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, int* err) {
  const bool ok = tma::mbar_wait(bar, parity, kWaitNs);
  if (__all_sync(0xffffffffu, ok)) return true;
  atomicExch(err, 1);
  return false;
}

// A compute warp's arrival: its words of the block are written.
__device__ __forceinline__ void arrive_done(uint64_t* bar, uint32_t lane) {
  tma::fence_proxy_async();
  __syncwarp();
  if (lane == 0) tma::mbar_arrive(bar);
}

}  // namespace wt

// The top strided pass of a network (layers [log n - 8, log n), one high block):
// BabyBear / KoalaBear plain sub-transforms, M31 per-block twiddles.
template <class F, bool DESC>
struct WPass {
  // rounds in execution order: forward 1, 0; inverse 0, 1
  static constexpr int RA = DESC ? 1 : 0, RB = 1 - RA;
  static constexpr wt::RowOrder kIn = DESC ? wt::kPlain : wt::kSwapped, kOut = DESC ? wt::kSwapped : wt::kPlain;
  static constexpr int kSmemBytes = wt::kRing * (int)kTileBytes + (int)(wt::kTabPairs * 8u) + (int)sizeof(wt::Bars);

  __device__ static void run(const CUtensorMap* min, const CUtensorMap* mout, const TmaArgs& a) {
    extern __shared__ __align__(1024) uint32_t smem_words[];
    uint32_t* ring = smem_words;
    uint2* tab = reinterpret_cast<uint2*>(ring + wt::kRing * kTileWords);
    wt::Bars* bars = reinterpret_cast<wt::Bars*>(tab + wt::kTabPairs);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    if (tid == 32 * wt::kWarps) {
      tma::prefetch_map(min);
      tma::prefetch_map(mout);
      wt::init_bars(bars);
    }
    wt::fill_table<F>(tab, a.tw, a.log_n, a.lo, 0, tid, wt::kThreads);
    __syncthreads();
    pdl_wait();
    if (warp == (uint32_t)wt::kWarps) {
      if (lane == 0)
        wt::producer(min, ring, bars, a, 1u, [&](uint32_t it, uint32_t, const uint32_t* src) {
          const wt::Coord c = wt::coord(a, blockIdx.x + it * gridDim.x);
          tma::store_5d(mout, (int32_t)(c.chunk << 5), 0, 0, 0, (int32_t)c.col, src);
        });
      return;
    }
    const wt::Lane l(warp, lane);
    uint32_t slot = 0, use = 0;
    for (uint32_t t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
      if (t + gridDim.x >= a.ntiles) pdl_trigger();  // the CTA's last tile
      uint32_t* buf = ring + slot * kTileWords;
      if (!wt::warp_wait(&bars->full[slot], use & 1u, a.err)) return;
      uint32_t v[32];
      wt::ld_io(buf, v, l);
      wt::round<F, DESC, RA>(v, tab, l.g);
      wt::exchange<RA>(buf, v, l);
      wt::round<F, DESC, RB>(v, tab, l.g);
      if (a.scale) {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = mul_shoup<F>(v[i], a.scale_w, a.scale_ws);
      } else if constexpr (!Net<F, DESC>::kGS) {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = reduce2p<F>(v[i]);
      }
      wt::st_io(buf, v, l);
      wt::arrive_done(&bars->done[slot], lane);
      if (++slot == (uint32_t)wt::kRing) { slot = 0; ++use; }
    }
  }
};

template <class F, bool DESC>
__global__ void __launch_bounds__(wt::kThreads, wt::kCtasPerSm)
warp_pass_kernel(const __grid_constant__ CUtensorMap min, const __grid_constant__ CUtensorMap mout, TmaArgs a) {
  WPass<F, DESC>::run(&min, &mout, a);
}

// Fused LDE middle step over M31 (TExpand's): inverse layers [lo, log_n), n^-1,
// then for every output block q the forward layers [lo, log_n) of the extended
// network with high block q.
struct WExpandM31 {
  using F = M31;
  static constexpr uint32_t kMaxQ = 4;
  static constexpr int kSmemBytes =
      wt::kRing * (int)kTileBytes + (int)((1u + kMaxQ) * wt::kTabPairs * 8u) + (int)sizeof(wt::Bars);

  __device__ static void run(const CUtensorMap* min, const CUtensorMap* mout, const TmaArgs& a) {
    extern __shared__ __align__(1024) uint32_t smem_words[];
    uint32_t* ring = smem_words;
    uint2* tabs = reinterpret_cast<uint2*>(ring + wt::kRing * kTileWords);  // inverse, then one per output block
    wt::Bars* bars = reinterpret_cast<wt::Bars*>(tabs + (1u + kMaxQ) * wt::kTabPairs);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t nq = 1u << a.log_q;
    if (tid == 32 * wt::kWarps) {
      tma::prefetch_map(min);
      tma::prefetch_map(mout);
      wt::init_bars(bars);
    }
    wt::fill_table<F>(tabs, a.tw, a.log_n, a.lo, 0, tid, wt::kThreads);
    for (uint32_t q = 0; q < nq; ++q)
      wt::fill_table<F>(tabs + (1u + q) * wt::kTabPairs, a.tw_fwd, a.log_n + a.log_q, a.lo, q, tid, wt::kThreads);
    __syncthreads();
    pdl_wait();
    if (warp == (uint32_t)wt::kWarps) {
      if (lane == 0)
        wt::producer(min, ring, bars, a, nq, [&](uint32_t it, uint32_t q, const uint32_t* src) {
          const wt::Coord c = wt::coord(a, blockIdx.x + it * gridDim.x);
          tma::store_5d(mout, (int32_t)(c.chunk << 5), 0, 0, (int32_t)q, (int32_t)c.col, src);
        });
      return;
    }
    const wt::Lane l(warp, lane);
    uint32_t slot = 0, use = 0;    // ring position of the next block
    uint32_t it = 0;
    for (uint32_t t = blockIdx.x; t < a.ntiles; t += gridDim.x, ++it) {
      if (t + gridDim.x >= a.ntiles) pdl_trigger();  // the CTA's last tile
      if (!wt::warp_wait(&bars->full[slot], (it / wt::kRing) & 1u, a.err)) return;
      uint32_t x[32];
      uint32_t* buf = ring + slot * kTileWords;
      wt::ld_io(buf, x, l);
      wt::round<F, false, 0>(x, tabs, l.g);
      wt::exchange<0>(buf, x, l);
      wt::round<F, false, 1>(x, tabs, l.g);
#pragma unroll
      for (int i = 0; i < 32; ++i) x[i] = mul_shoup<F>(x[i], a.scale_w, a.scale_ws);  // n^-1
      for (uint32_t q = 0; q < nq; ++q) {
        buf = ring + slot * kTileWords;
        // the buffer's previous block has left (block 0 sits where its tile arrived)
        if (q > 0 && use > 0 && !wt::warp_wait(&bars->empty[slot], (use - 1u) & 1u, a.err)) return;
        uint32_t v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = x[i];
        const uint2* tab = tabs + (1u + q) * wt::kTabPairs;
        wt::round<F, true, 1>(v, tab, l.g);
        wt::exchange<1>(buf, v, l);
        wt::round<F, true, 0>(v, tab, l.g);
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = reduce2p<F>(v[i]);
        wt::st_io(buf, v, l);
        wt::arrive_done(&bars->done[slot], lane);
        if (++slot == (uint32_t)wt::kRing) { slot = 0; ++use; }
      }
    }
  }
};

}  // namespace sfntt
