// layout.cu -- output conventions for LDE / NTT results (SoA batches).
//
// The transforms leave each column's rows in bit-reversed order, SoA
// (data[col * n + row]), as the reference does.  Two conventions used by the
// callers either side of the path:
//   * natural row order (Plonky3's coset_lde_batch returns natural-order rows):
//     out[col * n + r] = in[col * n + bitrev(r)];
//   * row-major rows, the input of Merkle commitment (one leaf per row):
//     out[R * batch + col] = in[col * n + r], R = r or bitrev(r).
// Both are pure permutations, HBM-bound: every word is read once and written
// once.  The reference's own permutation kernel is `bitrev_permute`
// (shaders/m31/m31_ntt_ct_dit_r2.metal:22-41), one word per thread.
//
// Kernels move tiles through shared memory so that global reads and writes are
// whole 128- to 512-byte segments:
//   bitrev_cols: tile (column, mid) holds words (hi << (L-5)) | (mid << 5) | lo
//     for hi, lo < 32; word (hi, mid, lo) goes to (rev5(lo), rev(mid), rev5(hi));
//     tiles mid and rev(mid) swap, so the permutation also runs in place.
//   transpose: tiles of columns x consecutive rows; each row of the tile
//     becomes consecutive words of one output row.
#include <algorithm>

#include "context.hpp"
#include "tma_launch.cuh"

namespace sfntt {
namespace {

constexpr int kLayoutThreads = 256;

__device__ __forceinline__ uint32_t rev_bits(uint32_t x, uint32_t bits) { return bits ? __brev(x) >> (32 - bits) : 0u; }

// log_n >= 10.  tiles = batch << (log_n - 10).  Tiles mid and rev(mid) of a
// column trade places, so one CTA handles the pair (the CTA of the larger mid
// skips): both are read before either is written, which also makes the
// permutation safe in place (in == out).
__global__ void __launch_bounds__(kLayoutThreads) bitrev_cols_kernel(const uint32_t* in, uint64_t in_stride,
                                                                     uint32_t* out, uint64_t out_stride,
                                                                     uint32_t log_n, uint64_t tiles) {
  __shared__ uint32_t ta[32][33], tb[32][33];
  const uint32_t mbits = log_n - 10;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t hi_shift = log_n - 5;
  for (uint64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const uint64_t col = t >> mbits;
    const uint32_t mid = (uint32_t)(t & ((1ull << mbits) - 1ull));
    const uint32_t rmid = rev_bits(mid, mbits);
    if (mid > rmid) continue;  // uniform over the CTA
    const uint32_t* sa = in + col * in_stride + ((uint64_t)mid << 5);
    const uint32_t* sb = in + col * in_stride + ((uint64_t)rmid << 5);
#pragma unroll
    for (uint32_t h = warp; h < 32; h += kLayoutThreads / 32) {
      ta[h][lane] = sa[((uint64_t)h << hi_shift) + lane];
      if (rmid != mid) tb[h][lane] = sb[((uint64_t)h << hi_shift) + lane];
    }
    __syncthreads();
    // tile mid's word (hi, lo) lands in tile rmid at row rev5(lo), word rev5(hi), and vice versa
    uint32_t* da = out + col * out_stride + ((uint64_t)rmid << 5);
    uint32_t* db = out + col * out_stride + ((uint64_t)mid << 5);
#pragma unroll
    for (uint32_t a = warp; a < 32; a += kLayoutThreads / 32) {
      const uint32_t hi = rev_bits(lane, 5), lo = rev_bits(a, 5);
      da[((uint64_t)a << hi_shift) + lane] = ta[hi][lo];
      if (rmid != mid) db[((uint64_t)a << hi_shift) + lane] = tb[hi][lo];
    }
    __syncthreads();
  }
}

// The same permutation on 64 x 64-word tiles (log_n >= 12): 256-byte global
// rows and 32 KB per CTA in flight.  The shared tile is XOR-swizzled, word
// (r, c) at r * 64 + (c ^ ((r >> 1) & 31)), so a row (fixed r) and the
// bit-reversed column read (rows rev6(j) for the 32 lanes j, whose r >> 1 are
// the 32 values rev5(j mod 32)) both touch 32 distinct banks.
constexpr int kWideThreads = 512;

__device__ __forceinline__ uint32_t swz64(uint32_t r, uint32_t c) { return r * 64u + (c ^ ((r >> 1) & 31u)); }

__global__ void __launch_bounds__(kWideThreads) bitrev_cols64_kernel(const uint32_t* in, uint64_t in_stride,
                                                                     uint32_t* out, uint64_t out_stride,
                                                                     uint32_t log_n, uint64_t tiles) {
  __shared__ uint32_t ta[64 * 64], tb[64 * 64];
  const uint32_t mbits = log_n - 12;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t hi_shift = log_n - 6;
  for (uint64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const uint64_t col = t >> mbits;
    const uint32_t mid = (uint32_t)(t & ((1ull << mbits) - 1ull));
    const uint32_t rmid = rev_bits(mid, mbits);
    if (mid > rmid) continue;  // uniform over the CTA
    const uint32_t* sa = in + col * in_stride + ((uint64_t)mid << 6);
    const uint32_t* sb = in + col * in_stride + ((uint64_t)rmid << 6);
#pragma unroll
    for (uint32_t h = warp; h < 64; h += kWideThreads / 32) {
#pragma unroll
      for (uint32_t w = lane; w < 64; w += 32) {
        ta[swz64(h, w)] = sa[((uint64_t)h << hi_shift) + w];
        if (rmid != mid) tb[swz64(h, w)] = sb[((uint64_t)h << hi_shift) + w];
      }
    }
    __syncthreads();
    // tile mid's word (hi, lo) lands in tile rmid at row rev6(lo), word rev6(hi), and vice versa
    uint32_t* da = out + col * out_stride + ((uint64_t)rmid << 6);
    uint32_t* db = out + col * out_stride + ((uint64_t)mid << 6);
#pragma unroll
    for (uint32_t a = warp; a < 64; a += kWideThreads / 32) {
      const uint32_t lo = rev_bits(a, 6);
#pragma unroll
      for (uint32_t j = lane; j < 64; j += 32) {
        const uint32_t hi = rev_bits(j, 6);
        da[((uint64_t)a << hi_shift) + j] = ta[swz64(hi, lo)];
        if (rmid != mid) db[((uint64_t)a << hi_shift) + j] = tb[swz64(hi, lo)];
      }
    }
    __syncthreads();
  }
}

// Row-major rows of up to 256 columns (log_n >= 5, 16-byte aligned buffers):
// tiles of every column x 32 kr rows, about 32 KiB.  TMA brings a tile in as
// 128-byte pieces, line = piece * batch + column, with the 128-byte swizzle; a
// lane then takes 4 consecutive rows of its column with one 128-bit load (lanes
// on consecutive columns: the swizzle spreads 8 of them over all banks) and
// writes them as four words of the row-major tile.  In row order that tile is
// one contiguous run of the output and leaves as one bulk copy, so a row of 400
// bytes costs no partial sectors; bit-reversed rows leave as one copy each
// (rows of whole 16-byte units) or by coalesced stores.  Bound by HBM (8 bytes
// per word; the reads are 128-byte runs megabytes apart); two input tiles per
// CTA keep the next load in flight.  Row order 2^19 x 100: 125 -> 70 us (6.0
// TB/s) against the 32 x 32 tiles, 2^21 x 256: 858 -> 756 us against the
// 128-column tiles, 2^20 x 7: 58 -> 25 us; bit-reversed 2^19 x 100: 144 -> 107
// us, 2^21 x 256: 873 -> 740 us.
constexpr uint32_t kRowsThreads = 256;
constexpr uint32_t kRowsMaxLines = 256;
struct RowsArgs {
  uint32_t* out;
  uint32_t log_n, batch;
  uint32_t lk;     // log2 of the 32-row pieces per tile
  uint32_t tiles;
  uint32_t bitrev;
  int* err;
};

__global__ void __launch_bounds__(kRowsThreads) transpose_tma_kernel(const __grid_constant__ CUtensorMap map_in,
                                                                     RowsArgs a) {
  extern __shared__ __align__(1024) uint32_t smem_rows[];
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t nb = a.batch, words = nb << (a.lk + 5);
  const uint32_t in_words = (words + 255u) & ~255u;  // 1024-byte aligned tiles (swizzle)
  uint32_t* ot = smem_rows + 2 * in_words;           // the row-major tile
  uint64_t* bar = reinterpret_cast<uint64_t*>(ot + in_words);
  uint32_t t = blockIdx.x;
  if (t >= a.tiles) return;
  auto load = [&](uint32_t tile, uint32_t buf) {
    tma::mbar_expect_tx(&bar[buf], words * 4u);
    tma::load_3d(smem_rows + buf * in_words, &map_in, 0, 0, (int32_t)(tile << a.lk), &bar[buf]);
  };
  if (tid == 0) {
    tma::prefetch_map(&map_in);
    tma::mbar_init(&bar[0], 1);
    tma::mbar_init(&bar[1], 1);
    tma::fence_mbar_init();
  }
  __syncthreads();
  if (tid == 0) load(t, 0);
  const uint32_t cgroups = (nb + 31u) >> 5;
  const uint32_t units = (cgroups << a.lk) * 8u;  // (piece, column group, 4-row chunk)
  for (uint32_t it = 0; t < a.tiles; t += gridDim.x, ++it) {
    const uint32_t buf = it & 1u;
    const uint32_t* it_in = smem_rows + buf * in_words;
    const uint32_t tn = t + gridDim.x;
    if (tid == 0 && tn < a.tiles) load(tn, buf ^ 1u);  // that buffer's readers passed the last barrier
    if (warp == 0) tma::wait_reads();                  // the previous tile's stores have read `ot`
    const bool ok = tma::mbar_wait(&bar[buf], (it >> 1) & 1u, kWaitNs);
    __syncthreads();
    for (uint32_t u = warp; u < units; u += kRowsThreads / 32) {
      const uint32_t j = u & 7u, pg = u >> 3;
      const uint32_t piece = pg / cgroups, col = ((pg - piece * cgroups) << 5) + lane;
      if (col < nb) {
        const uint32_t line = piece * nb + col;
        const uint4 q = *reinterpret_cast<const uint4*>(it_in + line * 32u + ((j ^ (line & 7u)) << 2));
        uint32_t* d = ot + (piece * 32u + j * 4u) * nb + col;
        d[0] = q.x;
        d[nb] = q.y;
        d[2 * nb] = q.z;
        d[3 * nb] = q.w;
      }
    }
    tma::fence_proxy_async();
    if (__syncthreads_or(!ok)) {
      if (tid == 0) {
        atomicExch(a.err, 1);
        if (tn < a.tiles) tma::mbar_wait(&bar[buf ^ 1u], ((it + 1) >> 1) & 1u, kWaitNs);
      }
      if (warp == 0) tma::wait_all();
      return;
    }
    const uint32_t r0 = t << (5 + a.lk);
    if (!a.bitrev) {
      if (tid == 0) {
        tma::store_bulk(a.out + (uint64_t)r0 * nb, ot, words * 4u);
        tma::commit();
      }
      continue;
    }
    // row i of the tile goes to output row bitrev(r0 + i) = bitrev(r0) + (bitrev(i) << ..)
    const uint32_t R0 = rev_bits(r0, a.log_n), sh = a.log_n - 5 - a.lk;
    if ((nb & 3u) == 0) {
      if (warp == 0) {
        for (uint32_t i = lane; i < (32u << a.lk); i += 32)
          tma::store_bulk(a.out + (uint64_t)(R0 + (rev_bits(i, 5 + a.lk) << sh)) * nb, ot + i * nb, nb * 4u);
        tma::commit();
      }
    } else {
      for (uint32_t i = warp; i < (32u << a.lk); i += kRowsThreads / 32) {
        uint32_t* d = a.out + (uint64_t)(R0 + (rev_bits(i, 5 + a.lk) << sh)) * nb;
        for (uint32_t c = lane; c < nb; c += 32) d[c] = ot[i * nb + c];
      }
    }
  }
  if (warp == 0) tma::wait_all();
}

// Row-major on 128-column x 32-row tiles (log_n >= 5, batch >= 128): 128-byte
// reads (32 rows of one column) and 512-byte writes (128 columns of one row),
// so a tile's output is 32 runs of 512 bytes, one per output row.  Tile word
// (column j, row i) at j * 33 + i: a column (fixed j, lanes over i) and a row
// (fixed i, lanes over j) both touch 32 distinct banks.
constexpr uint32_t kWideCols = 128;

__global__ void __launch_bounds__(kWideThreads) transpose_wide_kernel(const uint32_t* __restrict__ in,
                                                                      uint32_t* __restrict__ out, uint32_t log_n,
                                                                      uint32_t batch, uint32_t cblocks, uint32_t tiles,
                                                                      int bitrev) {
  __shared__ uint32_t tile[kWideCols * 33];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Loads: thread reads tile column warp + 16 q (q < 8) at row lane.  Stores:
  // thread writes tile row si + 4 q at column sj.  Addresses advance by
  // shifts from per-tile bases; a bit-reversed row r0 + i (r0 a multiple of
  // 32, i < 32) is rev(r0) + (rev5(i) << (log n - 5)).
  const uint32_t si = warp >> 2, sj = ((warp & 3u) << 5) + lane;
  for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const uint32_t rb = t / cblocks, cb = t - rb * cblocks;
    const uint32_t c0 = cb * kWideCols;
    const uint64_t r0 = (uint64_t)rb << 5;
    const uint32_t* src = in + ((uint64_t)(c0 + warp) << log_n) + r0 + lane;
#pragma unroll
    for (uint32_t q = 0; q < kWideCols / 16; ++q) {
      const uint32_t j = warp + 16u * q;
      if (c0 + j < batch) tile[j * 33 + lane] = __ldcs(src + ((uint64_t)q << (log_n + 4)));
    }
    __syncthreads();
    if (c0 + sj < batch) {
      uint32_t* dst = out + c0 + sj;
      if (bitrev) {
        const uint64_t rbase = (uint64_t)rev_bits((uint32_t)r0, log_n) + ((uint64_t)rev_bits(si, 5) << (log_n - 5));
        dst += rbase * batch;
        const uint64_t step = (uint64_t)batch << (log_n - 5);  // row rev5(4 q) << (log n - 5) = rev3(q) << (log n - 3)
#pragma unroll
        for (uint32_t q = 0; q < 8; ++q) __stcs(dst + (uint64_t)(rev_bits(4u * q, 5)) * step, tile[sj * 33 + si + 4u * q]);
      } else {
        dst += (r0 + si) * batch;
        const uint64_t step = 4ull * batch;
#pragma unroll
        for (uint32_t q = 0; q < 8; ++q) __stcs(dst + q * step, tile[sj * 33 + si + 4u * q]);
      }
    }
    __syncthreads();
  }
}

// Row-major rows of small batches and of buffers without 16-byte alignment:
// 32 x 32 tiles (log_n >= 5).  Tiles: ceil(batch / 32) column blocks x (n / 32) row blocks.
__global__ void __launch_bounds__(kLayoutThreads) transpose_kernel(const uint32_t* __restrict__ in,
                                                                   uint32_t* __restrict__ out, uint32_t log_n,
                                                                   uint32_t batch, uint32_t cblocks, uint64_t tiles,
                                                                   int bitrev) {
  __shared__ uint32_t tile[32][33];
  const uint64_t n = 1ull << log_n;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (uint64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const uint32_t cb = (uint32_t)(t % cblocks);
    const uint64_t r0 = (t / cblocks) << 5;
    const uint32_t c0 = cb << 5;
#pragma unroll
    for (uint32_t j = warp; j < 32; j += kLayoutThreads / 32)
      if (c0 + j < batch) tile[j][lane] = __ldcs(in + (uint64_t)(c0 + j) * n + r0 + lane);
    __syncthreads();
    const bool col_ok = c0 + lane < batch;
#pragma unroll
    for (uint32_t i = warp; i < 32; i += kLayoutThreads / 32) {
      const uint64_t r = r0 + i;
      const uint64_t R = bitrev ? rev_bits((uint32_t)r, log_n) : r;
      if (col_ok) __stcs(out + R * batch + c0 + lane, tile[lane][i]);
    }
    __syncthreads();
  }
}

// Natural row order of short columns (any size), in place or not: the thread
// owning row r <= bitrev(r) moves the pair.
__global__ void bitrev_pairs_kernel(const uint32_t* in, uint64_t in_stride, uint32_t* out, uint64_t out_stride,
                                    uint32_t log_n, uint64_t total) {
  const uint64_t mask = (1ull << log_n) - 1ull;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t c = i >> log_n, r = i & mask, rr = rev_bits((uint32_t)r, log_n);
    if (r <= rr) {
      const uint32_t x = in[c * in_stride + r], y = in[c * in_stride + rr];
      out[c * out_stride + rr] = x;
      out[c * out_stride + r] = y;
    }
  }
}

// Any shape (small columns): one word per thread.
__global__ void layout_words_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, uint32_t log_n,
                                    uint32_t batch, uint64_t total, int flags) {
  const uint64_t mask = (1ull << log_n) - 1ull;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t c = i >> log_n, r = i & mask;
    const uint64_t R = (flags & SFNTT_LAYOUT_NATURAL) ? rev_bits((uint32_t)r, log_n) : r;
    const uint64_t d = (flags & SFNTT_LAYOUT_ROW_MAJOR) ? R * batch + c : (c << log_n) + R;
    out[d] = in[i];
  }
}

uint32_t grid_for(const sfntt_ctx* ctx, uint64_t work) {
  return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(work, (uint64_t)ctx->sm_count * 8));
}

}  // namespace

Status bitrev_cols_dev(sfntt_ctx* ctx, const uint32_t* in, uint64_t in_stride, uint32_t* out, uint64_t out_stride,
                       uint32_t log_n, uint32_t batch, cudaStream_t s) {
  const uint64_t total = (uint64_t)batch << log_n;
  if (total == 0 || log_n == 0) {
    if (total && in != out) SFNTT_CU(cudaMemcpy2DAsync(out, out_stride * 4, in, in_stride * 4, 4, batch,
                                                       cudaMemcpyDeviceToDevice, s));
    return {};
  }
  launch_begin(ctx, s);
  if (log_n >= 12) {
    const uint64_t tiles = (uint64_t)batch << (log_n - 12);
    // 64 CTAs per SM, two resident: the CTAs in flight hold consecutive tiles,
    // whose 256-byte runs share DRAM rows (4 per SM, a stride of 4 x SMs
    // tiles between a CTA's tiles: 0.96 ms for the 2 GiB LDE output; 64: 0.76)
    const uint32_t grid = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(tiles, (uint64_t)ctx->sm_count * 64));
    bitrev_cols64_kernel<<<grid, kWideThreads, 0, s>>>(in, in_stride, out, out_stride, log_n, tiles);
    return launch_check(ctx, "layout_bitrev_cols", s, total * 8);
  }
  if (log_n >= 10) {
    const uint64_t tiles = (uint64_t)batch << (log_n - 10);
    bitrev_cols_kernel<<<grid_for(ctx, tiles), kLayoutThreads, 0, s>>>(in, in_stride, out, out_stride, log_n, tiles);
    return launch_check(ctx, "layout_bitrev_cols", s, total * 8);
  }
  bitrev_pairs_kernel<<<grid_for(ctx, (total + 255) / 256), 256, 0, s>>>(in, in_stride, out, out_stride, log_n, total);
  return launch_check(ctx, "layout_bitrev_pairs", s, total * 8);
}

// From how many words on bit-reversed rows of `batch` columns take the TMA tiles
// (us, register tiles and TMA tiles).  A row is a copy of its own, or words where
// it is no multiple of 16 bytes, so few columns never pay (2^20 x 64 137, 164).
// 65 to 72 and 129 to 144 columns leave four CTAs per SM, 73 to 96 and 145 to 192
// three, the others two, whose copies take longer to hide; and one column past
// 128 the register tiles are half empty.  2^16 x 72 10.7, 9.3, x 96 11.3, 11.5, x
// 128 11.1, 16.1, x 129 17.7, 14.1, x 250 28.2, 29.8, x 256 27.7, 24.3; 2^15 x 128
// 6.1, 8.9, x 129 9.7, 8.9, x 192 9.9, 8.6, x 250 11.4, 15.8; 2^17 x 73 21.4, 20.2, x
// 99 29.4, 34.1, x 128 27.8, 30.5; 2^18 x 99 63.7, 67.1, x 100 61.7, 55.2, x 127 72.7,
// 67.9; 2^19 x 99 143, 129.
uint64_t bitrev_rows_from(uint32_t batch) {
  const bool copies = (batch & 3u) == 0;
  if (batch < 72) return ~0ull;
  if (batch == 72 || (batch > 128 && batch <= 192)) return 1ull << 22;
  if (batch <= 96) return 1ull << 23;
  if (batch <= 128) return copies ? 3ull << 23 : 1ull << 25;
  return copies ? 3ull << 22 : 1ull << 24;
}

Status layout_dev(sfntt_ctx* ctx, const uint32_t* in, uint32_t* out, uint32_t log_n, uint32_t batch, int flags,
                  cudaStream_t s) {
  if (flags & ~(SFNTT_LAYOUT_NATURAL | SFNTT_LAYOUT_ROW_MAJOR)) return {SFNTT_INVALID_ARGUMENT, "unknown layout flags"};
  if (log_n > 31) return {SFNTT_INVALID_SIZE, "log_n > 31"};
  const uint64_t total = (uint64_t)batch << log_n;
  if (total == 0) return {};
  if (!in || !out) return {SFNTT_INVALID_ARGUMENT, "null buffer"};
  const bool natural = flags & SFNTT_LAYOUT_NATURAL;
  const bool rows = (flags & SFNTT_LAYOUT_ROW_MAJOR) && batch > 1;  // one column is its own row-major form
  const uintptr_t a = reinterpret_cast<uintptr_t>(in), b = reinterpret_cast<uintptr_t>(out);
  const bool same = a == b;
  if (!same && a < b + total * 4 && b < a + total * 4) return {SFNTT_INVALID_ARGUMENT, "layout buffers overlap"};
  if (same && rows) return {SFNTT_INVALID_ARGUMENT, "the row-major layout is out of place"};
  const uint64_t n = 1ull << log_n;
  if (!rows) {
    if (natural) return bitrev_cols_dev(ctx, in, n, out, n, log_n, batch, s);
    if (!same) SFNTT_CU(cudaMemcpyAsync(out, in, total * 4, cudaMemcpyDeviceToDevice, s));
    return {};
  }
  const char* name = natural ? "layout_transpose_bitrev" : "layout_transpose";
  // The TMA tiles pay from 2^22 words on (below, the launch and the first
  // tile's latency are the cost: 2^15 x 128 9.3 us here, 10.0 us there).  Above
  // 256 columns a tile no longer holds whole rows (2^19 x 301 in column blocks:
  // 333 us against 283 us).
  if (total >= (natural ? bitrev_rows_from(batch) : 1ull << 22) && batch <= kRowsMaxLines && log_n >= 5 &&
      aligned16(in) && aligned16(out)) {
    RowsArgs ra{};
    while (ra.lk < log_n - 5 && (batch << (ra.lk + 1)) <= kRowsMaxLines) ++ra.lk;
    ra.out = out; ra.log_n = log_n; ra.batch = batch; ra.bitrev = natural ? 1u : 0u;
    ra.tiles = 1u << (log_n - 5 - ra.lk);
    ra.err = ctx->err.as<int>();
    CUtensorMap map;
    const cuuint64_t dims[3] = {32, batch, n / 32}, strides[2] = {n * 4, 128};
    const cuuint32_t box[3] = {32, batch, 1u << ra.lk};
    SFNTT_TRY(tensor_map_encode(&map, in, 3, dims, strides, box, true));
    auto smem_of = [](uint32_t lines) { return (int)(3 * ((lines * 128 + 1023) & ~1023u)) + 16 + 1024; };
    const int smem = smem_of(batch << ra.lk);
    static std::atomic<uint64_t> smem_done{0};
    SFNTT_TRY(smem_limit_once(transpose_tma_kernel, smem_of(kRowsMaxLines), ctx->device, smem_done));
    const uint32_t per_sm = std::min<uint32_t>(8, 232448u / ((uint32_t)smem + 1024));
    const uint32_t grid = std::min<uint32_t>(ra.tiles, (uint32_t)ctx->sm_count * per_sm);
    launch_begin(ctx, s);
    transpose_tma_kernel<<<grid, kRowsThreads, smem, s>>>(map, ra);
    return launch_check(ctx, natural ? "layout_transpose_bitrev_tma" : "layout_transpose_tma", s, total * 8);
  }
  launch_begin(ctx, s);
  if (log_n >= 5 && batch >= kWideCols) {
    const uint32_t cblocks = (batch + kWideCols - 1) / kWideCols;
    const uint64_t tiles = (uint64_t)cblocks << (log_n - 5);  // batch * n / 4096 at most: < 2^29
    // 64 CTAs per SM, as the bit reversal (row-major 0.83 -> 0.80 ms on the 2 GiB LDE output)
    const uint32_t grid = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(tiles, (uint64_t)ctx->sm_count * 64));
    transpose_wide_kernel<<<grid, kWideThreads, 0, s>>>(in, out, log_n, batch, cblocks, (uint32_t)tiles,
                                                        natural ? 1 : 0);
    return launch_check(ctx, natural ? "layout_transpose_bitrev" : "layout_transpose", s, total * 8);
  }
  if (log_n >= 5) {
    const uint32_t cblocks = (batch + 31) / 32;
    const uint64_t tiles = (uint64_t)cblocks << (log_n - 5);
    transpose_kernel<<<grid_for(ctx, tiles), kLayoutThreads, 0, s>>>(in, out, log_n, batch, cblocks, tiles,
                                                                      natural ? 1 : 0);
    return launch_check(ctx, name, s, total * 8);
  }
  layout_words_kernel<<<grid_for(ctx, (total + 255) / 256), 256, 0, s>>>(in, out, log_n, batch, total, flags);
  return launch_check(ctx, "layout_words", s, total * 8);
}

}  // namespace sfntt
