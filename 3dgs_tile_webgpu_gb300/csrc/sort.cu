// Stable LSD radix sort pass over (uint32 key, uint32 value).
//
// Replaces the reference's 4-bit, 5-dispatch-per-pass radix sort
// (src/renderer/kernels/radix.ts:10-263, src/renderer/pipeline/RadixSorter.ts:50-322),
// which is a stable LSD sort; stability is the property the pass depends on
// (records enter in ordinal order for the depth sort and in depth-rank order
// for the tile sort, TiledGaussianPipeline.ts:144,442-446).
//
// One pass = reduce, scan, scatter with no look-back chain (a single-kernel
// decoupled look-back pass settles only a window of tiles per L2 round trip,
// which bounds it far below HBM speed on passes of tens of millions of keys).
// The items split into `chunks` contiguous runs of whole 4096-item tiles (one
// split, derived from the device-side count, shared by the two kernels; the
// runs differ by at most one tile, so that no SM gets two tiles more than
// another: with runs of ceil(tiles / chunks), 2.3M items kept 280 of the 456
// blocks busy):
//   k_chunk_count   keys of every (chunk, digit), by shared-memory atomics:
//                   a row of counts per chunk, and rows of sums over 16
//                   chunks each, added up by atomics;
//   k_chunk_scatter one block per chunk adds up the sums of the
//                   groups of chunks before its own and the rows before its
//                   own in its group (at most 29 + 15 rows; a kernel between
//                   the two that turned the counts into positions took 6 us a
//                   pass), then walks its tiles in order with running
//                   per-digit offsets: the keys of tile t+1 stream into
//                   shared memory by a bulk copy (cp.async.bulk, completion
//                   counted on an mbarrier) while tile t is ranked per digit
//                   within each warp (warp-striped layout: item j*32+lane of
//                   each warp's 512-item segment, so ranks follow index
//                   order), staged in place in block-sorted order, and
//                   written out with each digit's run contiguous; its values
//                   stream in while it is ranked.
// Stable: tiles in index order within a chunk, chunks in index order, ranks in
// index order within a tile.
// Bound by instructions and shared memory, not by HBM (2.4 TB/s at 398M
// records). The lanes of a digit are found by 8 ballots (95 instructions and 21
// shared-memory wavefronts per 32 items in all) or by each lane setting its bit
// in its digit's word (60 and 32): ballots alone keep the issue slots busy, the
// words alone the shared memory (73% of its wavefronts), so the rows of a
// warp take turns. us, depth sort of 6M items / of 2 x 17.5M, tile sort of
// 17.7M / 398M records: ballots 213 / 1099 / 230 / 5418, words 191 / 1083 / 211 /
// 5151, turns 191 / 1057 / 206 / 5028. Three of four rows by ballots 205 / 1080 /
// 218 / 5233. The tables leave no room for two value buffers; single buffers
// and 4 blocks per SM: 203 / 1119 / 224 / 5523; 512 threads of 8 items spill at 40
// registers (1201 for 2 x 17.5M).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "pass_common.cuh"

namespace gs {

constexpr int kCountWarps = kBlock / 32;
constexpr int kScatterThreads = 256;
constexpr int kSortWarps = kScatterThreads / 32;
constexpr int kSortItems = 16;  // kSortTile = 8 warps * 32 lanes * 16 items
static_assert(kSortTile == (uint32_t)(kScatterThreads * kSortItems), "a tile is 16 items per thread");

// Lanes of the warp holding the same BITS-bit digit, by ballot bit-splitting.
template <int BITS>
__device__ __forceinline__ uint32_t match_digit(uint32_t d, uint32_t valid_mask) {
  uint32_t peers = valid_mask;
#pragma unroll
  for (int b = 0; b < BITS; ++b) {
    const bool bit = (d >> b) & 1u;
    const uint32_t bal = __ballot_sync(0xffffffffu, bit);
    peers &= bit ? bal : ~bal;
  }
  return peers;
}

// Tiles [t0, t1) of chunk c when n items split over `chunks` chunks.
__device__ __forceinline__ void chunk_tiles(uint32_t n, uint32_t chunks, uint32_t c, uint32_t* t0, uint32_t* t1) {
  const uint32_t tiles = (uint32_t)(((uint64_t)n + kSortTile - 1) / kSortTile);
  *t0 = (uint32_t)((uint64_t)c * tiles / chunks);
  *t1 = (uint32_t)((uint64_t)(c + 1u) * tiles / chunks);
}

// A pass's digit of a key: BITS bits from `shift` on, of key - low for 9-bit
// digits.
template <int BITS>
__device__ __forceinline__ uint32_t digit_of(uint32_t key, uint32_t low, uint32_t shift) {
  return ((BITS > 8 ? key - low : key) >> shift) & ((1u << BITS) - 1u);
}

template <int BITS>
__global__ void __launch_bounds__(kBlock) k_chunk_count(const uint32_t* __restrict__ keys,
                                                        const uint32_t* __restrict__ n_ptr, uint32_t low,
                                                        uint32_t shift, uint32_t chunks,
                                                        uint32_t* __restrict__ counts, uint32_t* __restrict__ sums) {
  next_may_launch();
  constexpr uint32_t RADIX = 1u << BITS;
  __shared__ uint32_t s_hist[kCountWarps][RADIX];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  for (uint32_t i = tid; i < kCountWarps * RADIX; i += kBlock) (&s_hist[0][0])[i] = 0u;
  __syncthreads();
  const uint32_t n = *n_ptr;
  uint32_t t0, t1;
  chunk_tiles(n, chunks, blockIdx.x, &t0, &t1);
  const uint32_t begin = (uint32_t)min((uint64_t)t0 * kSortTile, (uint64_t)n);
  const uint32_t end = (uint32_t)min((uint64_t)t1 * kSortTile, (uint64_t)n);
  // Each warp takes 512-key runs: four 16-byte loads per lane in flight
  // before any counting (begin is a multiple of 4096, so they are aligned).
  constexpr uint32_t kRun = 512u;
  for (uint32_t s = begin + warp * kRun; s < end; s += kCountWarps * kRun) {
    uint32_t kk[16];
#pragma unroll
    for (uint32_t q = 0; q < 4u; ++q) {
      const uint32_t i0 = s + q * 128u + 4u * lane;
      if (i0 + 4u <= end) {
        const uint4 v = *reinterpret_cast<const uint4*>(keys + i0);
        kk[4 * q] = v.x; kk[4 * q + 1] = v.y; kk[4 * q + 2] = v.z; kk[4 * q + 3] = v.w;
      } else {
#pragma unroll
        for (uint32_t e = 0; e < 4u; ++e) kk[4 * q + e] = i0 + e < end ? keys[i0 + e] : 0u;
      }
    }
#pragma unroll
    for (uint32_t q = 0; q < 16u; ++q) {
      const bool ok = s + (q >> 2) * 128u + 4u * lane + (q & 3u) < end;
      const uint32_t d = digit_of<BITS>(kk[q], low, shift);
      const uint32_t d0 = __shfl_sync(0xffffffffu, d, 0);
      if (__all_sync(0xffffffffu, ok && d == d0)) {
        if (lane == 0u) atomicAdd(&s_hist[warp][d0], 32u);
      } else if (ok) {
        atomicAdd(&s_hist[warp][d], 1u);
      }
    }
  }
  __syncthreads();
  for (uint32_t d = tid; d < RADIX; d += kBlock) {
    uint32_t sum = 0;
#pragma unroll
    for (int w = 0; w < kCountWarps; ++w) sum += s_hist[w][d];
    counts[(size_t)blockIdx.x * RADIX + d] = sum;
    if (sum) atomicAdd(sums + blockIdx.x / kSumChunks * kSumWords + d, sum);
  }
}

// Two buffers of keys, one of values: the keys of tile t+1 stream in while
// tile t is ranked and scattered, its values while it is ranked.
constexpr size_t kChunkDynSmem = 3 * kSortTile * sizeof(uint32_t);

// Digits owned by a thread of the scatter.
__host__ __device__ constexpr int digits_per_thread(int bits) { return bits > 8 ? 2 : 1; }

template <int BITS>
struct ScatterShared {
  uint16_t warp_hist[kSortWarps][1u << BITS];  // a warp's items per digit, then its first tile position
  uint32_t match[kSortWarps][1u << BITS];  // lanes of the warp's current row holding each digit; zero in between
  uint32_t delta[1u << BITS];  // global position of the tile's item i of a digit, minus i
  uint32_t scan[8];
  unsigned long long bar[3];  // bulk-copy completion of the two key buffers and the value buffer
};

// Exclusive scan of one value per digit over the threads below 256, in two
// block barriers; every thread of the block calls it.
__device__ __forceinline__ uint32_t digit_scan(uint32_t v, uint32_t* s_scan) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31u && warp < 8u) s_scan[warp] = x;
  __syncthreads();
  uint32_t before = 0;
#pragma unroll
  for (uint32_t w = 0; w < 7u; ++w) before += w < warp ? s_scan[w] : 0u;
  return before + x - v;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Bulk copy of one tile's keys or values (items base .. min(base + 4096, n))
// into buf, issued by thread 0 and counted on the mbarrier; the last n % 4
// items of a ragged tile (a bulk copy moves whole 16-byte units) come by plain
// loads, visible after the next block barrier.
__device__ __forceinline__ void load_tile_bulk(const uint32_t* __restrict__ in, uint32_t base, uint32_t n,
                                               uint32_t* buf, uint32_t bar) {
  const uint32_t items = min(kSortTile, n - base);
  const uint32_t whole = items & ~3u;  // items moved by the bulk copy
  if (threadIdx.x == 0) {
    const uint32_t bytes = whole * 4u;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    if (bytes) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the buffer's previous reads come first
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       smem_addr(buf)),
                   "l"(in + base), "r"(bytes), "r"(bar)
                   : "memory");
    }
  }
  for (uint32_t e = whole + threadIdx.x; e < items; e += kScatterThreads) buf[e] = in[base + e];
}

// Bounded wait for phase `parity` of the mbarrier (about a second of polls).
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity) {
  uint32_t backoff = 16;
  for (uint32_t polls = 0; polls < kSpinLimit; ++polls) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    __nanosleep(backoff);
    backoff = backoff < 256 ? backoff * 2 : 256;
  }
  return false;
}

// Ranks the tile held in kb/vb (items base .. base + 4096, those below n),
// stages it in place in block-sorted order and writes each digit's run to its
// global position. FULL: every item of the tile is below n. `run`: the global
// position of the next item of digit threadIdx.x (threads below 2^BITS).
// Leaves warp_hist zeroed and run advanced past the tile. parity: the phase of
// the value buffer's barrier; false if the values never landed.
template <int BITS, bool FULL>
__device__ __forceinline__ bool scatter_tile(ScatterShared<BITS>& sm, uint32_t* kb, uint32_t* vb, uint32_t base,
                                             uint32_t n, uint32_t low, uint32_t shift,
                                             uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
                                             uint32_t (&run)[digits_per_thread(BITS)], uint32_t parity) {
  constexpr uint32_t RADIX = 1u << BITS;
  constexpr int D = digits_per_thread(BITS);
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t wofs = warp * 32u * kSortItems;  // warp-striped: item j*32+lane of the warp's segment
  uint32_t k[kSortItems], rank[kSortItems];
#pragma unroll
  for (int j = 0; j < kSortItems; ++j) k[j] = kb[wofs + (uint32_t)j * 32u + lane];
#pragma unroll
  for (int j = 0; j < kSortItems; ++j) {
    const bool ok = FULL || base + wofs + (uint32_t)j * 32u + lane < n;
    const uint32_t valid = FULL ? 0xffffffffu : __ballot_sync(0xffffffffu, ok);
    const uint32_t d = digit_of<BITS>(k[j], low, shift);
    uint32_t peers = valid;
    if (!FULL || (j & 1)) {
      peers = match_digit<BITS>(d, valid);
    } else if (!__all_sync(0xffffffffu, d == __shfl_sync(0xffffffffu, d, 0))) {
      // Each lane sets its bit in its digit's word; one digit for the whole
      // row would serialise the 32 atomics and needs none.
      atomicOr(&sm.match[warp][d], 1u << lane);
      __syncwarp();
      peers = sm.match[warp][d];
    }
    const uint32_t before = __popc(peers & lt);
    uint32_t cnt = 0;
    if (ok) cnt = sm.warp_hist[warp][d];
    rank[j] = cnt + before;
    __syncwarp();
    if (ok && before == 0) {
      sm.warp_hist[warp][d] = (uint16_t)(cnt + __popc(peers));
      if (FULL && !(j & 1)) sm.match[warp][d] = 0u;
    }
    __syncwarp();
  }
  __syncthreads();

  // Thread d: the tile's items of digit d (of digits 2d and 2d + 1 where there
  // are more digits than threads), and with the digits below it the tile
  // position of each warp's first item of the digit (one look-up per item
  // below).
  const bool owns = tid * D < RADIX;
  if constexpr (D == 1) {
    uint32_t count = 0;
    if (owns) {
#pragma unroll
      for (int w = 0; w < kSortWarps; ++w) count += sm.warp_hist[w][tid];
    }
    uint32_t at = digit_scan(count, sm.scan);
    if (owns) {
      sm.delta[tid] = run[0] - at;
      run[0] += count;
#pragma unroll
      for (int w = 0; w < kSortWarps; ++w) {
        const uint32_t c = sm.warp_hist[w][tid];
        sm.warp_hist[w][tid] = (uint16_t)at;
        at += c;
      }
    }
  } else {
    // Both digits in the halves of a word (no sum of a tile passes 16 bits):
    // half the shared accesses and half the spills of two counters per thread
    // (6M items, three passes: 178 -> 163 us).
    uint32_t count = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) count += reinterpret_cast<const uint32_t*>(sm.warp_hist[w])[tid];
    const uint32_t low_count = count & 0xffffu, first = digit_scan(low_count + (count >> 16), sm.scan);
    reinterpret_cast<uint2*>(sm.delta)[tid] = make_uint2(run[0] - first, run[1] - (first + low_count));
    run[0] += low_count;
    run[1] += count >> 16;
    uint32_t at = first | (first + low_count) << 16;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
      uint32_t& word = reinterpret_cast<uint32_t*>(sm.warp_hist[w])[tid];
      const uint32_t c = word;
      word = at;
      at += c;
    }
  }
  __syncthreads();

  // Keys first (every raw key is in registers), then the values (read raw
  // into the keys' registers, then written once every thread has read).
#pragma unroll
  for (int j = 0; j < kSortItems; ++j) {
    if (FULL || base + wofs + (uint32_t)j * 32u + lane < n) {
      const uint32_t d = digit_of<BITS>(k[j], low, shift);
      rank[j] += sm.warp_hist[warp][d];
      kb[rank[j]] = k[j];
    }
  }
  const bool landed = bar_wait(smem_addr(&sm.bar[2]), parity);
#pragma unroll
  for (int j = 0; j < kSortItems; ++j) k[j] = vb[wofs + (uint32_t)j * 32u + lane];
  if (!__syncthreads_and(landed)) return false;
#pragma unroll
  for (int j = 0; j < kSortItems; ++j)
    if (FULL || base + wofs + (uint32_t)j * 32u + lane < n) vb[rank[j]] = k[j];
  __syncthreads();

  const uint32_t items = FULL ? kSortTile : min(kSortTile, n - base);
#pragma unroll 4
  for (uint32_t i = tid; i < items; i += kScatterThreads) {
    const uint32_t key = kb[i];
    const uint32_t dst = sm.delta[digit_of<BITS>(key, low, shift)] + i;
    keys_out[dst] = key;
    vals_out[dst] = vb[i];
  }
  for (uint32_t i = tid; i < kSortWarps * RADIX * sizeof(uint16_t) / 4u; i += kScatterThreads)
    reinterpret_cast<uint32_t*>(&sm.warp_hist[0][0])[i] = 0u;
  __syncthreads();
  return true;
}

template <int BITS>
__global__ void __launch_bounds__(kScatterThreads, kChunkBlocksPerSm)
    k_chunk_scatter(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                    uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
                    const uint32_t* __restrict__ n_ptr, uint32_t low, uint32_t shift, uint32_t chunks,
                    const uint32_t* __restrict__ counts, const uint32_t* __restrict__ sums,
                    uint32_t* __restrict__ spare, uint32_t* __restrict__ err) {
  after_previous();
  constexpr uint32_t RADIX = 1u << BITS;
  constexpr int D = digits_per_thread(BITS);
  __shared__ __align__(16) ScatterShared<BITS> sm;
  extern __shared__ uint4 s_dyn[];
  uint32_t* s_buf = reinterpret_cast<uint32_t*>(s_dyn);

  const uint32_t tid = threadIdx.x, c = blockIdx.x;
  // The other sums, used by the pass before this one, start the next at zero.
  if (c < sum_rows(chunks))
    for (uint32_t i = tid; i < kSumWords; i += kScatterThreads) spare[c * kSumWords + i] = 0u;
  const uint32_t n = *n_ptr;
  uint32_t t0, t1;
  chunk_tiles(n, chunks, c, &t0, &t1);
  if (t0 >= t1) return;
  if (tid < 3u) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sm.bar[tid])) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  uint32_t phases = 0;  // parity of the next phase of each buffer's barrier
  uint32_t* vb = s_buf + 2u * kSortTile;
  load_tile_bulk(keys_in, t0 * kSortTile, n, s_buf, smem_addr(&sm.bar[0]));
  for (uint32_t i = tid; i < kSortWarps * RADIX; i += kScatterThreads) (&sm.match[0][0])[i] = 0u;
  for (uint32_t i = tid; i < kSortWarps * RADIX * sizeof(uint16_t) / 4u; i += kScatterThreads)
    reinterpret_cast<uint32_t*>(&sm.warp_hist[0][0])[i] = 0u;
  // Thread d: the chunk's first position of its digits: keys of the digits
  // below, and of the digit itself in the chunks before.
  const uint32_t group = c / kSumChunks, groups = sum_rows(chunks);
  uint32_t all[D] = {}, run[D] = {}, sum = 0;
  if (tid * D < RADIX) {
    // The thread's digits of row `row` of a table of rows of `words` words.
    auto digits = [&](const uint32_t* table, uint32_t row, uint32_t words, uint32_t (&x)[D]) {
      const uint32_t* at = table + (size_t)row * words + tid * D;
      if constexpr (D == 2) {
        const uint2 q = *reinterpret_cast<const uint2*>(at);
        x[0] = q.x;
        x[1] = q.y;
      } else {
        x[0] = *at;
      }
    };
#pragma unroll 8
    for (uint32_t g = 0; g < groups; ++g) {
      uint32_t x[D];
      digits(sums, g, kSumWords, x);
#pragma unroll
      for (int i = 0; i < D; ++i) {
        all[i] += x[i];
        run[i] += g < group ? x[i] : 0u;
      }
    }
#pragma unroll
    for (uint32_t r = 0; r < kSumChunks - 1u; ++r) {
      const uint32_t row = group * kSumChunks + r;
      uint32_t x[D] = {};
      if (row < c) digits(counts, row, RADIX, x);
#pragma unroll
      for (int i = 0; i < D; ++i) run[i] += x[i];
    }
  }
#pragma unroll
  for (int i = 0; i < D; ++i) sum += all[i];
  uint32_t below = digit_scan(sum, sm.scan);
#pragma unroll
  for (int i = 0; i < D; ++i) {
    run[i] += below;
    below += all[i];
  }

  for (uint32_t t = t0; t < t1; ++t) {
    const uint32_t k = (t - t0) & 1u, base = t * kSortTile;
    uint32_t* kb = s_buf + k * kSortTile;
    load_tile_bulk(vals_in, base, n, vb, smem_addr(&sm.bar[2]));
    if (t + 1u < t1)
      load_tile_bulk(keys_in, base + kSortTile, n, s_buf + (k ^ 1u) * kSortTile, smem_addr(&sm.bar[k ^ 1u]));
    bool ok = __syncthreads_and(bar_wait(smem_addr(&sm.bar[k]), (phases >> k) & 1u));
    const uint32_t parity = (t - t0) & 1u;
    if (ok) {
      if ((uint64_t)base + kSortTile <= n)
        ok = scatter_tile<BITS, true>(sm, kb, vb, base, n, low, shift, keys_out, vals_out, run, parity);
      else
        ok = scatter_tile<BITS, false>(sm, kb, vb, base, n, low, shift, keys_out, vals_out, run, parity);
    } else {
      bar_wait(smem_addr(&sm.bar[2]), parity);
    }
    phases ^= 1u << k;
    if (!ok) {
      // A copy never landed: flag the frame and leave, after the copy of the
      // next keys (if one was issued) had its own bounded wait.
      if (tid == 0) atomicOr(err, 4u);
      if (t + 1u < t1) bar_wait(smem_addr(&sm.bar[k ^ 1u]), (phases >> (k ^ 1u)) & 1u);
      return;
    }
  }
}

template <int B>
void launch_chunk_bits(uint32_t chunks, const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out,
                       uint32_t* vals_out, const uint32_t* n_ptr, uint32_t low, uint32_t shift, uint32_t* counts,
                       uint32_t* sums, uint32_t* spare, uint32_t* err, cudaStream_t st) {
  k_chunk_count<B><<<chunks, kBlock, 0, st>>>(keys_in, n_ptr, low, shift, chunks, counts, sums);
  launch_after(k_chunk_scatter<B>, chunks, kScatterThreads, kChunkDynSmem, st, keys_in, vals_in, keys_out, vals_out,
               n_ptr, low, shift, chunks, counts, sums, spare, err);
}

template <int B>
void configure_bits() {
  cudaFuncSetAttribute(k_chunk_scatter<B>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kChunkDynSmem);
}

void prepare_sort_kernels() {
  configure_bits<1>(); configure_bits<2>(); configure_bits<3>(); configure_bits<4>();
  configure_bits<5>(); configure_bits<6>(); configure_bits<7>(); configure_bits<8>();
  configure_bits<9>();
}

uint32_t chunk_pass_chunks(uint32_t n_max, int sms) {
  const uint64_t tiles = ((uint64_t)n_max + kSortTile - 1) / kSortTile;
  return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(tiles, (uint64_t)kChunkBlocksPerSm * (uint64_t)sms));
}

void launch_chunk_pass(int bits, const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out,
                       uint32_t* vals_out, const uint32_t* n_ptr, uint32_t low, int shift, uint32_t chunks,
                       uint32_t* counts, uint32_t* sums, uint32_t* spare, uint32_t* err, cudaStream_t st) {
#define GS_CHUNK(B)                                                                                               \
  case B:                                                                                                         \
    launch_chunk_bits<B>(chunks, keys_in, vals_in, keys_out, vals_out, n_ptr, low, (uint32_t)shift, counts, sums, \
                         spare, err, st);                                                                         \
    break;
  switch (bits) {
    GS_CHUNK(1)
    GS_CHUNK(2)
    GS_CHUNK(3)
    GS_CHUNK(4)
    GS_CHUNK(5)
    GS_CHUNK(6)
    GS_CHUNK(7)
    GS_CHUNK(9)
    default:
      GS_CHUNK(8)
  }
#undef GS_CHUNK
}

}  // namespace gs
