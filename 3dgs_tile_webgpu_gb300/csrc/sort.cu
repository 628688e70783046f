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
#include "radix.cuh"

namespace gs {

constexpr int kSortItems = 16;  // kSortTile = 8 warps * 32 lanes * 16 items
static_assert(kSortTile == (uint32_t)(kScatterThreads * kSortItems), "a tile is 16 items per thread");

// A pass's digit of a key: BITS bits from `shift` on, of key - low for 9-bit
// digits.
template <int BITS>
struct PassDigit {
  uint32_t low, shift;
  __device__ __forceinline__ uint32_t operator()(uint32_t key) const {
    return ((BITS > 8 ? key - low : key) >> shift) & ((1u << BITS) - 1u);
  }
};

template <int BITS>
__global__ void __launch_bounds__(kBlock) k_chunk_count(const uint32_t* __restrict__ keys,
                                                        const uint32_t* __restrict__ n_ptr, uint32_t low,
                                                        uint32_t shift, uint32_t chunks,
                                                        uint32_t* __restrict__ counts, uint32_t* __restrict__ sums) {
  next_may_launch();
  constexpr uint32_t RADIX = 1u << BITS;
  __shared__ uint32_t s_hist[kCountWarps][RADIX];
  const uint32_t tid = threadIdx.x;
  for (uint32_t i = tid; i < kCountWarps * RADIX; i += kBlock) (&s_hist[0][0])[i] = 0u;
  __syncthreads();
  const uint32_t n = *n_ptr;
  uint32_t t0, t1;
  chunk_tiles(n, kSortTile, chunks, blockIdx.x, &t0, &t1);
  const uint32_t begin = (uint32_t)min((uint64_t)t0 * kSortTile, (uint64_t)n);
  const uint32_t end = (uint32_t)min((uint64_t)t1 * kSortTile, (uint64_t)n);
  count_keys<BITS>(s_hist, keys, begin, end, PassDigit<BITS>{low, shift});
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
  __shared__ unsigned long long s_bar[3];  // bulk-copy completion of the two key buffers and the value buffer
  extern __shared__ uint4 s_dyn[];
  uint32_t* s_buf = reinterpret_cast<uint32_t*>(s_dyn);

  const uint32_t tid = threadIdx.x, c = blockIdx.x;
  // The other sums, used by the pass before this one, start the next at zero.
  if (c < sum_rows(chunks))
    for (uint32_t i = tid; i < kSumWords; i += kScatterThreads) spare[c * kSumWords + i] = 0u;
  const uint32_t n = *n_ptr;
  uint32_t t0, t1;
  chunk_tiles(n, kSortTile, chunks, c, &t0, &t1);
  if (t0 >= t1) return;
  if (tid < 3u) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&s_bar[tid])) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  uint32_t phases = 0;  // parity of the next phase of each buffer's barrier
  uint32_t* vb = s_buf + 2u * kSortTile;
  load_tile_bulk(keys_in, t0 * kSortTile, n, s_buf, smem_addr(&s_bar[0]));
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
    load_tile_bulk(vals_in, base, n, vb, smem_addr(&s_bar[2]));
    if (t + 1u < t1)
      load_tile_bulk(keys_in, base + kSortTile, n, s_buf + (k ^ 1u) * kSortTile, smem_addr(&s_bar[k ^ 1u]));
    bool ok = __syncthreads_and(bar_wait(smem_addr(&s_bar[k]), (phases >> k) & 1u));
    const uint32_t parity = (t - t0) & 1u;
    if (ok) {
      const PassDigit<BITS> digit = {low, shift};
      auto landed = [&] { return bar_wait(smem_addr(&s_bar[2]), parity); };
      if ((uint64_t)base + kSortTile <= n)
        ok = scatter_tile<BITS, kSortItems, true>(sm, kb, vb, base, n, digit, keys_out, vals_out, run, landed);
      else
        ok = scatter_tile<BITS, kSortItems, false>(sm, kb, vb, base, n, digit, keys_out, vals_out, run, landed);
    } else {
      bar_wait(smem_addr(&s_bar[2]), parity);
    }
    phases ^= 1u << k;
    if (!ok) {
      // A copy never landed: flag the frame and leave, after the copy of the
      // next keys (if one was issued) had its own bounded wait.
      if (tid == 0) atomicOr(err, kErrorCopy);
      if (t + 1u < t1) bar_wait(smem_addr(&s_bar[k ^ 1u]), (phases >> (k ^ 1u)) & 1u);
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
