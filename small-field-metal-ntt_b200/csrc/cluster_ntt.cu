// cluster_ntt.cu -- one-launch NTT of columns of 2^13 .. 2^16 points on a
// thread-block cluster.
//
// A column of n = 2^(12+X) points is split over the CTAs of one cluster, CTA r
// owning the contiguous positions [r 2^B, (r+1) 2^B) in shared memory (B = 12: 2
// to 16 CTAs of 256 threads, 16 being the non-portable size; B = 13: 1 to 8 of
// 512).  Layers [0, 12) pair positions inside a block and run on the tile
// engine's rounds (TPass<F, DESC, Kind::C, 12>: registers, shared-memory
// exchanges).  The X cross layers [12, 12+X) pair positions 2^12 apart: the
// points {base + k 2^12 : k < 2^X} (base < 2^12) form one group, one or two
// points per block, and each thread owns 16 / 2^X whole groups, so these layers
// run in registers.  The exchange between the two parts goes through distributed
// shared memory.
//
//   inverse (layers ascending): load the block, in-block layers, cluster
//     barrier, gather the groups from the cluster's blocks, cross layers and
//     n^-1, store the groups (consecutive threads own consecutive bases:
//     coalesced); a second cluster barrier, split around the last two steps,
//     keeps every block alive until the others have read it.
//   forward (layers descending): load the groups, cross layers, scatter them
//     into the owning blocks, cluster barrier, in-block layers, store the block.
//
// Every global read of a column happens before the cluster's first barrier and
// every global write after it, so the transform works in place.
//
// One column is a chain of latencies: 16 layers on the SMs of one cluster, the
// twiddles' L2 latency and the launch.  Blocks of 2^12 words halve the work per
// SM of 2^13-word ones, and the twiddles -- BabyBear / KoalaBear's in-block table
// into shared memory, M31's 32 KiB of per-block twiddles into L1, the cross
// twiddles into registers -- are fetched before the wait for the previous kernel
// (programmatic dependent launch), so they overlap its end.  Forward / inverse of
// one column from a graph, 2^13-word blocks with the twiddles fetched layer by
// layer -> now: BabyBear 2^13 6.7 / 7.1 -> 4.0 / 4.5 us, 2^16 7.9 / 8.4 -> 5.0 /
// 5.3 us; M31 2^13 6.1 / 6.0 -> 4.1 / 4.4 us, 2^16 7.2 / 7.4 -> 5.4 / 5.3 us.
// Batches that fill the SMs take the wider blocks in places, launched plainly
// and with the cross twiddles read layer by layer (see cluster_form).
#include <cooperative_groups.h>

#include "context.hpp"
#include "pdl.cuh"
#include "tile_tma.cuh"

namespace sfntt {
namespace {

namespace cg = cooperative_groups;

// B: log2 of a block's words, 12 or 13.
template <class F, bool DESC, int X, int B>
struct ClusterNtt {
  static_assert(B == 12 || B == 13, "blocks of 2^12 or 2^13 words");
  using TP = TPass<F, DESC, Kind::C, 12, false, false, false, false, B == 12 ? 12 : 0>;
  static constexpr int PPB = 1 << (B - 12);  // points of a cross group per block
  static constexpr int CS = (1 << X) / PPB;  // CTAs per column
  static constexpr int G = 1 << X;           // points per cross group
  static constexpr int GPT = 16 / G;         // groups per thread
  static constexpr uint32_t NT = TP::NT;
  static constexpr uint32_t LOG_N = 12 + X;
  static constexpr uint32_t BASES = 4096u / CS;  // group bases per CTA
  static_assert(NT == (B == 12 ? 256 : 512) && TP::E == 16 && BASES == GPT * NT && TP::TWORDS == 1u << B,
                "one thread: 16 points in whole groups");

  // Butterflies of one group and layer j, low points in order: cross_at(k, j)
  // numbers the twiddles a thread needs for one group (M31: 2^(X-1-j) per layer,
  // the same for every group; BabyBear / KoalaBear: 2^j).
  static constexpr int CT = G - 1;  // per group
  static constexpr int CN = F::kMontgomery ? GPT * CT : CT;
  __device__ static constexpr int cross_at(int k, int j) {
    return F::kMontgomery ? ((1 << j) - 1) + (k & ((1 << j) - 1)) : (G - (G >> j)) + (k >> (j + 1));
  }

  // Twiddle of the cross butterfly whose lower point is k (bit j clear) of the
  // group at `base`, layer L = 12 + j: BabyBear / KoalaBear tw[L][pos mod 2^L],
  // M31 tw[L][pos >> (L+1)] (the same for every base).
  // A volatile load stays ahead of the wait for the previous kernel.
  __device__ static __forceinline__ uint2 ld_tw(const uint2* p) {
    uint2 r;
    asm volatile("ld.global.nc.v2.u32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(p));
    return r;
  }
  __device__ static __forceinline__ const uint2* cross_at_mem(const uint2* tw, uint32_t base, int k, int j) {
    const uint32_t L = 12u + (uint32_t)j;
    if constexpr (F::kMontgomery) {
      return tw + ((1u << L) - 1u) + base + ((uint32_t)(k & ((1 << j) - 1)) << 12);
    } else {
      const uint32_t n = 1u << LOG_N;
      return tw + (n - (n >> L)) + ((uint32_t)k >> (j + 1));
    }
  }

  // Every cross twiddle of the thread's groups, all loads in flight at once.
  __device__ static __forceinline__ void load_cross(uint2 (&t)[CN], uint32_t base0, const uint2* tw) {
#pragma unroll
    for (int gi = 0; gi < (F::kMontgomery ? GPT : 1); ++gi)
#pragma unroll
      for (int j = 0; j < X; ++j)
#pragma unroll
        for (int k = 0; k < G; ++k) {
          if (k & (1 << j)) continue;
          const int first = F::kMontgomery ? (k & ((1 << j) - 1)) : ((k >> (j + 1)) << (j + 1));
          if (k == first) t[gi * CT + cross_at(k, j)] = ld_tw(cross_at_mem(tw, base0 + (uint32_t)gi * NT, k, j));
        }
  }

  // The X cross layers on the thread's groups (forward: descending, inverse:
  // ascending, then n^-1); canonical values out.  B = 13: twiddles from memory.
  __device__ static __forceinline__ void cross(uint32_t (&v)[16], const uint2 (&t)[CN], uint32_t base0, const uint2* tw,
                                               uint32_t scale_w, uint32_t scale_ws) {
#pragma unroll
    for (int gi = 0; gi < GPT; ++gi) {
#pragma unroll
      for (int jj = 0; jj < X; ++jj) {
        const int j = DESC ? (X - 1 - jj) : jj;
#pragma unroll
        for (int k = 0; k < G; ++k) {
          if (k & (1 << j)) continue;
          uint2 w;
          if constexpr (B == 12) w = t[(F::kMontgomery ? gi * CT : 0) + cross_at(k, j)];
          else w = __ldg(cross_at_mem(tw, base0 + (uint32_t)gi * NT, k, j));
          butterfly<F, DESC>(v[gi * G + k], v[gi * G + (k | (1 << j))], w);
        }
      }
    }
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      if constexpr (!DESC) v[m] = mul_shoup<F>(v[m], scale_w, scale_ws);
      else if constexpr (!Net<F, true>::kGS) v[m] = reduce2p<F>(v[m]);  // lazy CT values to [0, p)
    }
  }

  __device__ static void run(uint32_t* d, const uint2* tw, uint32_t scale_w, uint32_t scale_ws) {
    extern __shared__ __align__(1024) uint32_t smem_words[];
    uint32_t* tile = smem_words;                                // the block, in TP's swizzled layout
    uint2* tws = reinterpret_cast<uint2*>(tile + TP::TWORDS);  // the block's twiddles, layers [0, 12)
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank();
    const uint32_t tid = threadIdx.x;
    const uint64_t n = 1ull << LOG_N;
    uint32_t* col = d + (uint64_t)(blockIdx.x / CS) * n;
    TmaArgs a{};
    a.tw = tw;
    a.log_n = LOG_N;
    a.lo = 0;
    a.batch = 1;
    a.log_tpc = (uint32_t)(LOG_N - B);
    if constexpr (TP::kRound0Copy) a.tw0 = tw + n;  // M31 tables with n >= 2^13 carry it
    TileCoord g{};
    g.pos_base = rank << B;
    const uint32_t base0 = rank * BASES + tid;  // group gi: base0 + gi NT
    uint2 ctw[CN];
    // The tables do not depend on the previous kernel: under programmatic
    // dependent launch their loads overlap its end.
    pdl_trigger();
    if constexpr (TP::kStaged) {
      TP::stage_twiddles(tws, tw, tid);
    } else if constexpr (B == 12) {
      // layers 0..7 of the block are 255 lines of 128 bytes, one per thread;
      // the last thread takes layer 8's 64 bytes and what follows them
      const uint32_t L = tid < 255u ? 7u - (31u - __clz(255u - tid)) : 8u;
      const char* p = reinterpret_cast<const char*>(tw + (n - (n >> L)) + (g.pos_base >> (L + 1)) +
                                                    16u * (tid - (256u - (256u >> L))));
#pragma unroll
      for (uint32_t i = 0; i < 128u; i += 32u) {  // its four sectors
        uint32_t word;
        asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(word) : "l"(p + i));
      }
    }
    if constexpr (B == 12) load_cross(ctw, base0, tw);
    pdl_wait();
    uint32_t v[16];
    if constexpr (DESC) {
      // Distributed shared memory may be written only once every block of the
      // cluster is known to run: arrive here, wait just before the first
      // remote store, so the barrier overlaps the loads and cross layers.
      asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
#pragma unroll
      for (int gi = 0; gi < GPT; ++gi)
#pragma unroll
        for (int k = 0; k < G; ++k) v[gi * G + k] = col[base0 + (uint32_t)gi * NT + ((uint32_t)k << 12)];
      cross(v, ctw, base0, tw, 0u, 0u);
      asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
#pragma unroll
      for (int gi = 0; gi < GPT; ++gi)
#pragma unroll
        for (int k = 0; k < G; ++k) {
          uint32_t* owner = cluster.map_shared_rank(tile, (unsigned)(k / PPB));
          owner[TP::sw(base0 + (uint32_t)gi * NT + ((uint32_t)(k % PPB) << 12))] = v[gi * G + k];
        }
      cluster.sync();  // every block complete (and the staged twiddles visible)
      TP::template ld<TP::kFirst>(tile, v, tid);
      TP::template rounds<0>(tile, v, a, tws, g, tid);
      TP::finish(v, a, g, tid);
      TP::template st<TP::kLast>(tile, v, tid);
      __syncthreads();
      uint4* out = reinterpret_cast<uint4*>(col + g.pos_base);
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i) {
        const uint32_t c = 4u * (tid + i * NT);
        out[c >> 2] = *reinterpret_cast<const uint4*>(tile + TP::sw(c));
      }
    } else {
      const uint4* in = reinterpret_cast<const uint4*>(col + g.pos_base);
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i) {
        const uint32_t c = 4u * (tid + i * NT);
        *reinterpret_cast<uint4*>(tile + TP::sw(c)) = in[c >> 2];  // sw keeps 16-byte runs together
      }
      __syncthreads();
      TP::template ld<TP::kFirst>(tile, v, tid);
      TP::template rounds<0>(tile, v, a, tws, g, tid);
      TP::finish(v, a, g, tid);
      TP::template st<TP::kLast>(tile, v, tid);
      cluster.sync();  // every block complete
#pragma unroll
      for (int gi = 0; gi < GPT; ++gi)
#pragma unroll
        for (int k = 0; k < G; ++k) {
          const uint32_t* owner = cluster.map_shared_rank(tile, (unsigned)(k / PPB));
          v[gi * G + k] = owner[TP::sw(base0 + (uint32_t)gi * NT + ((uint32_t)(k % PPB) << 12))];
        }
      // No block may leave while another still reads it: arrive once the
      // reads are performed (release), wait only before leaving, so the
      // barrier overlaps the cross layers and the stores.
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
      cross(v, ctw, base0, tw, scale_w, scale_ws);
#pragma unroll
      for (int gi = 0; gi < GPT; ++gi)
#pragma unroll
        for (int k = 0; k < G; ++k) col[base0 + (uint32_t)gi * NT + ((uint32_t)k << 12)] = v[gi * G + k];
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
  }
};

template <class F, bool DESC, int X, int B>
__global__ void __launch_bounds__(ClusterNtt<F, DESC, X, B>::NT, B == 12 ? 3 : 1)
cluster_ntt_kernel(uint32_t* d, const uint2* tw, uint32_t scale_w, uint32_t scale_ws) {
  ClusterNtt<F, DESC, X, B>::run(d, tw, scale_w, scale_ws);
}

template <class F, bool DESC, int X, int B>
Status launch_cluster(sfntt_ctx* ctx, uint32_t* d, uint32_t batch, const uint2* tw, uint32_t scale_w, bool early,
                      cudaStream_t s) {
  using C = ClusterNtt<F, DESC, X, B>;
  constexpr int smem = 4 * (int)C::TP::TWORDS + 8 * (int)C::TP::TW_ENTRIES + 1024;
  auto kern = cluster_ntt_kernel<F, DESC, X, B>;
  static std::atomic<uint64_t> smem_done{0};
  if (C::CS > 8 && !(smem_done.load(std::memory_order_acquire) & (1ull << (ctx->device & 63))))
    SFNTT_CU(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  SFNTT_TRY(smem_limit_once(kern, smem, ctx->device, smem_done));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(batch * (uint32_t)C::CS);
  cfg.blockDim = dim3(C::NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)C::CS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
#ifdef SFNTT_NO_PDL
  cfg.numAttrs = 1;
#else
  cfg.numAttrs = early ? 2 : 1;
#endif
  const uint32_t scale_ws = (uint32_t)(((uint64_t)scale_w << 32) / F::P);
  launch_begin(ctx, s);
  SFNTT_CU(cudaLaunchKernelEx(&cfg, kern, d, tw, scale_w, scale_ws));
  static const std::string name = std::string(F::kTag) + (DESC ? "_fwd" : "_inv") + "_cluster" +
                                  std::to_string(C::CS) + (B == 13 ? "w" : "");
  return launch_check(ctx, name.c_str(), s, ((uint64_t)batch << C::LOG_N) * 8u);
}

// Clusters of 2^13-word blocks that run at once with one CTA per SM.
template <class F, bool DESC, int X>
uint32_t wide_clusters(const sfntt_ctx* ctx) {
  using C = ClusterNtt<F, DESC, X, 13>;
  static std::atomic<int> known[64];  // per device: clusters + 1
  std::atomic<int>& k = known[ctx->device & 63];
  if (const int n = k.load(std::memory_order_relaxed)) return (uint32_t)(n - 1);
  auto kern = cluster_ntt_kernel<F, DESC, X, 13>;
  constexpr int more_than_half = 116 << 10;  // of an SM's shared memory
  static std::atomic<uint64_t> smem_done{0};
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)C::CS);
  cfg.blockDim = dim3(C::NT);
  cfg.dynamicSmemBytes = more_than_half;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)C::CS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (!smem_limit_once(kern, more_than_half, ctx->device, smem_done).ok() ||
      cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  k.store(n + 1, std::memory_order_relaxed);
  return (uint32_t)n;
}

// Block size and launch of a batch, by blocks of 2^12 words per SM (us per call
// in a graph of calls: 2^12-word blocks launched early, plainly, 2^13-word blocks).
//   BabyBear / KoalaBear: up to 0.76, 2^12 early (2^14 x 18 4.2, 6.9, 7.2; 2^16 x 4
// 4.7, 7.4, 8.1).  Above, CTAs launched early pack onto the SMs that come free
// first, and without that two of them on an SM lose to one of 2^13 words as long
// as each of those has an SM (2^14 x 41 8.5, 8.5, 7.3; 2^15 x 27 9.3, 9.1, 8.0; 2^16
// x 15 10.0, 10.9, 8.3), but for the inverse of 2^16 points (x 10 6.9, 9.9, 9.0; x 15
// 9.1, 11.8, 9.1).  Then 2^12 early again (2^15 x 36 9.7, 10.3, 10.9; inverse 9.3,
// 11.6, 15.6).  2^13 points: only batches that 2^12 early suits come here.
//   M31, whose twiddles come through L1: early up to 0.24 (2^16 x 1 4.8, 5.2, 6.8),
// plainly up to 1.4 (2^15 x 5 5.5, 4.9, 7.0; 2^14 x 24 7.7, 4.8, 6.7; 2^16 x 12 9.3, 7.5, 7.5), wide while
// each has an SM (2^14 x 74 8.5, 8.6, 6.9), then early (2^15 x 37 9.0, 8.8, 13);
// pairs that divide evenly early (2^13 x 148 6.0, 6.4, 6.7).
// On several streams the forms differ by a tenth (8 streams, 2^14 x 55 4.0, 4.0,
// 3.7), but for M31 around 1.4 (2^16 x 12 4.1 against 5.4 with wide blocks).
struct ClusterForm { bool wide, early; };
template <class F, bool DESC, int X>
constexpr bool kMayBeWide = !F::kMontgomery || (X > 1 && (X < 4 || DESC));
template <class F, bool DESC, int X>
ClusterForm cluster_form(const sfntt_ctx* ctx, uint32_t batch) {
  const uint64_t sms = (uint64_t)ctx->sm_count, blocks = (uint64_t)batch << X;
  if constexpr (!kMayBeWide<F, DESC, X>) {
    return {false, true};
  } else {
    const bool wide = blocks <= 2 * sms && batch <= wide_clusters<F, DESC, X>(ctx);
    if (F::kMontgomery) return {wide && 25 * blocks > 19 * sms, !wide || 25 * blocks <= 19 * sms};
    if (X == 1 && blocks % sms == 0) return {false, true};
    if (5 * blocks <= 7 * sms) return {false, 25 * blocks <= 6 * sms};
    return {wide, !wide};
  }
}

template <class F, bool DESC, int X>
Status launch_blocks(sfntt_ctx* ctx, uint32_t* d, uint32_t batch, const uint2* tw, uint32_t scale_w, cudaStream_t s) {
  const ClusterForm f = cluster_form<F, DESC, X>(ctx, batch);
  if constexpr (kMayBeWide<F, DESC, X>) {
    if (f.wide) return launch_cluster<F, DESC, X, 13>(ctx, d, batch, tw, scale_w, f.early, s);
  }
  return launch_cluster<F, DESC, X, 12>(ctx, d, batch, tw, scale_w, f.early, s);
}

template <class F, bool DESC>
Status cluster_dispatch(sfntt_ctx* ctx, uint32_t* d, uint32_t log_n, uint32_t batch, const uint2* tw,
                        uint32_t scale_w, cudaStream_t s) {
  switch (log_n) {
    case 13: return launch_blocks<F, DESC, 1>(ctx, d, batch, tw, scale_w, s);
    case 14: return launch_blocks<F, DESC, 2>(ctx, d, batch, tw, scale_w, s);
    case 15: return launch_blocks<F, DESC, 3>(ctx, d, batch, tw, scale_w, s);
    case 16: return launch_blocks<F, DESC, 4>(ctx, d, batch, tw, scale_w, s);
    default: return {SFNTT_INVALID_ARGUMENT, "cluster NTT: 2^13 .. 2^16 points"};
  }
}

}  // namespace

// Against the passes (forward + inverse, us, passes and clusters).  BabyBear /
// KoalaBear: 2^13 points are one pass, so the clusters take what they start early
// without packing, up to 5/8 blocks of 2^12 words per SM and whole waves of up to
// three (x 46 10.3, 9.3; x 74 10.5, 8.8; x 120 10.9, 15.1); longer columns up to
// three per SM (2^14 x 41 18.3, 15.4; x 100 20.2, 19.0; 2^15 x 50 25.2, 23.1; 2^16 x
// 24 25.5, 24.8; x 31 26.1, 26.9).
//   M31's passes read their twiddles from L2 or stage them per tile, so it wins
// longer.  A pass takes two tiles of 2^13 words per SM and round, a round filled or
// not, the clusters a time that grows with the batch: up to where each of the
// first rounds is about three quarters full, in the fourth where it has just begun
// (2^14 x 148 23.7, 28.8; x 172 37.2, 30.3; x 296 37.8, 46.0; 2^15 x 111 46.0, 41.3;
// x 222 58.5, 71.9; 2^13 x 592 35.1, 39.9; x 641 48.6, 43.3).  2^16 points 3.1
// blocks per SM (x 24 28.8, 25.4; x 28 29.1, 27.0; x 33 29.2, 31.0).
//   The last batch of each range, whole waves, stays on the clusters, where it has
// been since they were built (2^16 x 37 BabyBear 26.2, 34.8; M31 2^14 x 592 65.9, 83.6).
bool cluster_ntt_fits(const sfntt_ctx* ctx, int field, uint32_t log_n, uint32_t batch, const void* d) {
  if (ctx->no_cluster || log_n < 13 || log_n > 16 || batch == 0) return false;
  if ((reinterpret_cast<uintptr_t>(d) & 15u) != 0) return false;
  const uint64_t blocks = (uint64_t)batch << (log_n - 12), sms = (uint64_t)ctx->sm_count;
  const uint64_t last = (log_n == 16 ? 4 : is_monty(field) ? 3 : 16) * sms;
  if (blocks >= last) return blocks == last;
  if (log_n == 16) return 10 * blocks <= 31 * sms;
  if (is_monty(field)) return log_n > 13 || 8 * blocks <= 5 * sms || blocks % sms == 0;
  const uint64_t rounds = (blocks + 4 * sms - 1) / (4 * sms);
  const uint64_t tenths = rounds == 4 ? 31 : log_n == 14 ? 30 : log_n == 15 ? 34 : 33;  // blocks per SM and round
  return 10 * blocks <= tenths * rounds * sms;
}

Status cluster_ntt_dev(sfntt_ctx* ctx, int field, bool inverse, uint32_t* d, uint32_t log_n, uint32_t batch,
                       const uint2* tw, uint32_t scale_w, cudaStream_t s) {
  return with_field(field, [&](auto f) -> Status {
    using F = decltype(f);
    return inverse ? cluster_dispatch<F, false>(ctx, d, log_n, batch, tw, scale_w, s)
                   : cluster_dispatch<F, true>(ctx, d, log_n, batch, tw, scale_w, s);
  });
}

}  // namespace sfntt
