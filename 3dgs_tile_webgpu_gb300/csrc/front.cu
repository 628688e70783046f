// The fused front of small launches: everything of the pass before the
// rasterizer (projection, visibility compaction, depth sort, intersection
// scan, emission, tile sort, tile ranges, raster work list) in one cooperative
// kernel whose blocks meet at grid barriers, instead of 23-26 kernels.
//
// Why: a launch of up to a few hundred thousand ordinals keeps each of those
// kernels busy for 2-5 us, below the cost of a launch (about 4 us of host time
// and 2-5 us of ramp-up and drain on the GPU each); a grid barrier costs
// 1-2 us. Whole frames at 1280x720, separate kernels / front: 2000 splats 118 /
// 61 us, 60k 137 / 86, 200k 188 / 151 (pipeline.cu: kFrontMaxItems).
//
// Every buffer ends up with the same contents as after the separate kernels.
// What differs is how the stages split the work:
//  * Compaction: the projection leaves the number of visible items of each 32
//    (a byte); a block sums the bytes before its units.
//  * Sorts of up to 2048 items run in one block, without barriers.
//  * Sort passes: up to a tile per block, a block ranks its tile, publishes its
//    256 digit counts, and after a barrier sums the rows before its own; above
//    that a run of tiles per block, counted, and scattered after the barrier
//    (chunk_pass). The depth sort
//    sorts key - (smallest visible key), and passes whose digit no key has are
//    left out (an LSD pass over equal digits moves nothing): the start buffer
//    is chosen so that the result lands where the host expects it.
//  * Scan: a block sums its ranks' tile counts, and after a barrier adds up
//    the sums of the blocks before it.
// Data that one block writes and another reads goes through plain loads
// (never the non-coherent path) after a barrier's acquire.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>

#include "emission.cuh"
#include "pass_common.cuh"
#include "projection.cuh"
#include "radix.cuh"

namespace gs {

namespace {

constexpr int kFrontWarps = kBlock / 32;
constexpr uint32_t kRadix = 256;  // digits of a pass (8 bits; narrower tile digits use the first ones)

// A sort tile of kBlock * IPT items: digit counts of each warp, then the tile
// in digit order on its way out.
template <int IPT>
struct TileShared {
  uint32_t warp_hist[kFrontWarps][kRadix];
  uint32_t excl[kRadix];  // tile position of each digit's first item
  uint32_t run[kRadix];   // global position of the chunk's next item of each digit
  uint32_t keys[kBlock * IPT], vals[kBlock * IPT];
};

struct ProjectShared {
  float snorm[256];
  uint32_t group;
  CountShared count;
};

// The chunked passes': two buffers of keys, one of values, and the tables of a
// tile.
constexpr int kChunkItems = 8;
constexpr uint32_t kChunkTile = kScatterThreads * kChunkItems;
struct ChunkShared {
  uint32_t keys[2][kChunkTile], vals[kChunkTile];
  ScatterShared<8> scatter;
};

union FrontShared {
  ProjectShared project;
  TileShared<4> tile4;
  TileShared<8> tile8;
  ChunkShared chunk;
  EmitShared emit;
};

// Meets the other blocks that arrive at this counter: waits until it reads
// `target`. The counters start at zero with the launch's staged batch table.
// Bounded: false (for all threads of the block) when `limit` polls saw some
// block missing.
__device__ __forceinline__ bool grid_barrier(uint32_t* counter, uint32_t target, uint32_t limit) {
  __syncthreads();
  bool ok = true;
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
    uint32_t seen, polls = 0;
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
      if (seen >= target) break;
      if (++polls >= limit) {
        ok = false;
        break;
      }
      if (polls > 64u) __nanosleep(polls > 4096u ? 256 : 32);
    }
  }
  return __syncthreads_and(ok);
}

// Block-wide sum of one value per thread (in every thread).
__device__ __forceinline__ unsigned long long block_sum(unsigned long long v, unsigned long long* s_warp) {
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  __syncthreads();
  if ((threadIdx.x & 31u) == 0u) s_warp[threadIdx.x >> 5] = v;
  __syncthreads();
  unsigned long long sum = 0;
#pragma unroll
  for (int w = 0; w < kFrontWarps; ++w) sum += s_warp[w];
  return sum;
}

// One sort pass's parameters: digit = ((key - low) >> shift) & mask.
struct Pass {
  const uint32_t* keys_in;
  const uint32_t* vals_in;
  uint32_t* keys_out;
  uint32_t* vals_out;
  uint32_t n, low, shift, mask;
  uint32_t* counts;  // a row of 256 per block
  uint32_t* sums;    // sums of kSumRows rows each, zero on entry
  uint32_t* spare;   // the same of the next pass, to be zeroed
  uint32_t* barrier; // the sort's own barrier counter
  __device__ __forceinline__ uint32_t digit(uint32_t key) const { return ((key - low) >> shift) & mask; }
};

// Loads the tile at `base` (warp-striped: item j * 32 + lane of the warp's
// segment, so ranks follow index order) and ranks its items per digit; leaves
// warp_hist holding each warp's first position within its digit, excl the
// tile position of each digit, and returns (thread d < 256) the tile's count
// of digit d.
template <int IPT>
__device__ __forceinline__ uint32_t rank_tile(TileShared<IPT>& sm, uint32_t* s_scan, const Pass& p, uint32_t base,
                                              uint32_t (&k)[IPT], uint32_t (&v)[IPT], uint32_t (&rank)[IPT]) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u, first = base + warp * 32u * IPT + lane;
#pragma unroll
  for (int j = 0; j < IPT; ++j) {
    k[j] = first + 32u * j < p.n ? p.keys_in[first + 32u * j] : 0u;
    v[j] = first + 32u * j < p.n ? p.vals_in[first + 32u * j] : 0u;
  }
  for (uint32_t i = tid; i < kFrontWarps * kRadix; i += kBlock) (&sm.warp_hist[0][0])[i] = 0u;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < IPT; ++j) {
    const bool ok = first + 32u * j < p.n;
    const uint32_t valid = __ballot_sync(0xffffffffu, ok);
    const uint32_t d = p.digit(k[j]);
    const uint32_t peers = match_digit<8>(d, valid);
    const uint32_t before = __popc(peers & lt);
    uint32_t cnt = 0;
    if (ok) cnt = sm.warp_hist[warp][d];
    rank[j] = cnt + before;
    __syncwarp();
    if (ok && before == 0) sm.warp_hist[warp][d] = cnt + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  uint32_t count = 0;
#pragma unroll
  for (int w = 0; w < kFrontWarps; ++w) {
    const uint32_t c = sm.warp_hist[w][tid];
    sm.warp_hist[w][tid] = count;
    count += c;
  }
  uint32_t total;
  sm.excl[tid] = block_exclusive_scan<false>(count, s_scan, &total);
  return count;
}

// Puts the ranked tile into shared memory in digit order.
template <int IPT>
__device__ __forceinline__ void arrange_tile(TileShared<IPT>& sm, const Pass& p, uint32_t base,
                                             const uint32_t (&k)[IPT], const uint32_t (&v)[IPT],
                                             const uint32_t (&rank)[IPT]) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t first = base + warp * 32u * IPT + lane;
  __syncthreads();  // excl, run and warp_hist are complete
#pragma unroll
  for (int j = 0; j < IPT; ++j) {
    if (first + 32u * j < p.n) {
      const uint32_t d = p.digit(k[j]);
      const uint32_t at = rank[j] + sm.excl[d] + sm.warp_hist[warp][d];
      sm.keys[at] = k[j];
      sm.vals[at] = v[j];
    }
  }
  __syncthreads();
}

// Writes the ranked tile out, each digit's items from run[digit] on.
template <int IPT>
__device__ __forceinline__ void write_tile(TileShared<IPT>& sm, const Pass& p, uint32_t base,
                                           const uint32_t (&k)[IPT], const uint32_t (&v)[IPT],
                                           const uint32_t (&rank)[IPT]) {
  const uint32_t tid = threadIdx.x;
  arrange_tile<IPT>(sm, p, base, k, v, rank);
  const uint32_t count = min((uint32_t)(kBlock * IPT), p.n - base);
#pragma unroll 4
  for (uint32_t i = tid; i < count; i += kBlock) {
    const uint32_t key = sm.keys[i], d = p.digit(key);
    const uint32_t dst = sm.run[d] + (i - sm.excl[d]);
    p.keys_out[dst] = key;
    p.vals_out[dst] = sm.vals[i];
  }
}

// Rows of the sums of a grid's count rows.
__host__ __device__ __forceinline__ uint32_t front_sum_rows(uint32_t grid) { return (grid + 15u) / 16u; }

// The kernel's arguments.
struct Front {
  BatchView b;
  PassOptions o;
  float4 *mean, *conic, *color, *rec, *erec;
  uint32_t *tile_counts, *keys, *vis_off, *dk0, *dk1, *dv0, *dv1, *ordered, *ioff, *tk0, *tk1, *tv0, *tv1;
  uint32_t *tile_offsets, *tile_order;  // tile_order null: tiles rasterize in tile order
  uint32_t* scratch;                    // a count row (256 words) per block, then twice the sums' rows
  Control* ctl;
  uint32_t* frame;         // the staged batch table's frame parameters (FrameParam)
  uint32_t* output_state;
  uint32_t capacity;
  uint32_t tile_passes, digit_bits;
  uint32_t small_sort;     // most items of a pass over tiles of 1024
  uint32_t limit;          // polls of a barrier before it expires
  uint32_t withhold;       // test hook: block 0 leaves before the compaction
};

// Rows summed up in one row of sums: a block adds the sums of the groups
// before its own and the rows of its group, at most grid / 16 + 15 rows in all.
constexpr uint32_t kSumRows = 16;

// The global position of row c's first item of digit tid: the items of the
// digits below, of all rows, and of the digit in the rows before.
__device__ __forceinline__ uint32_t first_position(const Pass& p, uint32_t* s_scan, uint32_t c, uint32_t groups) {
  const uint32_t tid = threadIdx.x, group = c / kSumRows;
  uint32_t all = 0, before = 0, total;
#pragma unroll 8
  for (uint32_t g = 0; g < groups; ++g) {
    const uint32_t x = p.sums[g * kRadix + tid];
    all += x;
    before += g < group ? x : 0u;
  }
#pragma unroll
  for (uint32_t r = 0; r < kSumRows - 1u; ++r) {
    const uint32_t row = group * kSumRows + r;
    before += row < c ? p.counts[row * kRadix + tid] : 0u;
  }
  return block_exclusive_scan<false>(all, s_scan, &total) + before;
}

// A pass with one tile of kBlock * IPT items for each of the first blocks:
// ranks stay in registers over the barrier. The other blocks take no part;
// they wait at the grid's next barrier (a barrier of 98 blocks takes 0.8 us,
// of 391 2 us). `last`: that barrier follows, so the pass ends without one.
template <int IPT>
__device__ __forceinline__ bool tile_pass(TileShared<IPT>& sm, uint32_t* s_scan, const Pass& p, uint32_t* round,
                                          bool last, uint32_t limit) {
  const uint32_t tid = threadIdx.x, c = blockIdx.x;
  const uint32_t rows = (p.n + kBlock * IPT - 1u) / (kBlock * IPT), groups = (rows + kSumRows - 1u) / kSumRows;
  if (c >= rows) return true;
  uint32_t k[IPT], v[IPT], rank[IPT];
  const uint32_t count = rank_tile<IPT>(sm, s_scan, p, c * kBlock * IPT, k, v, rank);
  p.counts[c * kRadix + tid] = count;
  if (count) atomicAdd(p.sums + c / kSumRows * kRadix + tid, count);
  if (!grid_barrier(p.barrier, ++*round * rows, limit)) return false;
  if (c < groups) p.spare[c * kRadix + tid] = 0u;
  sm.run[tid] = first_position(p, s_scan, c, groups);
  write_tile<IPT>(sm, p, c * kBlock * IPT, k, v, rank);
  return last || grid_barrier(p.barrier, ++*round * rows, limit);
}

// Asynchronous copies of the warp's own 256 items of the tile at base (those
// below n) into buf, 16 bytes each. They go through L2, which holds what other
// blocks wrote before the last barrier.
__device__ __forceinline__ void load_segment(uint32_t* buf, const uint32_t* in, uint32_t base, uint32_t n) {
  const uint32_t lane = threadIdx.x & 31u, first = (threadIdx.x >> 5) * 32u * kChunkItems + 4u * lane;
#pragma unroll
  for (uint32_t q = 0; q < kChunkItems / 4u; ++q) {
    const uint32_t i = first + q * 128u;
    if (base + i >= n) continue;
    const uint32_t bytes = min(n - base - i, 4u) * 4u;  // the rest of the 16 becomes zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(buf + i)),
                 "l"(in + base + i), "r"(bytes)
                 : "memory");
  }
}
// Ends a group of copies; waits for all but the last `PENDING` groups.
__device__ __forceinline__ void end_copies() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void wait_copies() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
  __syncwarp();  // the warp reads what its other lanes copied
}

// A pass over more items than a tile of 2048 per block: each block takes a
// contiguous run of 2048-item tiles, counts its digits, and after a barrier
// scatters the tiles as sort.cu's kernels do (radix.cuh: the keys of the next
// tile and the values are on their way while a tile is ranked). Tiles of 4096
// items take 62 KB of tables instead of 37, which the other stages miss as L1,
// and 16 items per thread spill: 300k splats at 1001x563 269 instead of 264 us,
// 390k at 1280x720 (1.5M records) 261 instead of 251. Frames of n splats, M
// records, us, with tiles whose loads were waited for and positions from a third
// barrier / so: 100k at 1280x720, 1.2M 201 / 160; 390k, 4.7M 443 / 370; 200k at
// 1920x1080, 23M 994 / 833; 20k at 3840x2160, 20M 1452 / 1181.
__device__ __forceinline__ bool chunk_pass(ChunkShared& sm, uint32_t* s_scan, const Pass& p, uint32_t* round, bool last,
                                           uint32_t limit) {
  const uint32_t tid = threadIdx.x, c = blockIdx.x, groups = front_sum_rows(gridDim.x);
  const auto digit = [&](uint32_t key) { return p.digit(key); };
  uint32_t t0, t1;
  chunk_tiles(p.n, kChunkTile, gridDim.x, c, &t0, &t1);
  uint32_t(*hist)[kRadix] = sm.scatter.match;  // the counts' histograms; zero again afterwards
  for (uint32_t i = tid; i < kFrontWarps * kRadix; i += kBlock) (&hist[0][0])[i] = 0u;
  for (uint32_t i = tid; i < kFrontWarps * kRadix / 2u; i += kBlock)
    reinterpret_cast<uint32_t*>(&sm.scatter.warp_hist[0][0])[i] = 0u;
  __syncthreads();
  count_keys<8>(hist, p.keys_in, (uint32_t)min((uint64_t)t0 * kChunkTile, (uint64_t)p.n),
                (uint32_t)min((uint64_t)t1 * kChunkTile, (uint64_t)p.n), digit);
  __syncthreads();
  uint32_t count = 0;
#pragma unroll
  for (int w = 0; w < kFrontWarps; ++w) {
    count += hist[w][tid];
    hist[w][tid] = 0u;
  }
  p.counts[c * kRadix + tid] = count;
  if (count) atomicAdd(p.sums + c / kSumRows * kRadix + tid, count);
  if (!grid_barrier(p.barrier, ++*round * gridDim.x, limit)) return false;
  if (c < groups) p.spare[c * kRadix + tid] = 0u;
  if (t0 < t1) {
    load_segment(sm.keys[0], p.keys_in, t0 * kChunkTile, p.n);
    end_copies();
    uint32_t run[1] = {first_position(p, s_scan, c, groups)};
    for (uint32_t t = t0; t < t1; ++t) {
      const uint32_t k = (t - t0) & 1u, base = t * kChunkTile;
      load_segment(sm.vals, p.vals_in, base, p.n);
      end_copies();
      if (t + 1u < t1) load_segment(sm.keys[k ^ 1u], p.keys_in, base + kChunkTile, p.n);
      end_copies();
      wait_copies<2>();  // the tile's keys
      const auto landed = [] {
        wait_copies<1>();  // its values
        return true;
      };
      if ((uint64_t)base + kChunkTile <= p.n)
        scatter_tile<8, kChunkItems, true>(sm.scatter, sm.keys[k], sm.vals, base, p.n, digit, p.keys_out, p.vals_out,
                                           run, landed);
      else
        scatter_tile<8, kChunkItems, false>(sm.scatter, sm.keys[k], sm.vals, base, p.n, digit, p.keys_out, p.vals_out,
                                            run, landed);
    }
  }
  return last || grid_barrier(p.barrier, ++*round * gridDim.x, limit);
}

// A sort of at most one tile of 2048 items (block 0 alone): the items stay in
// shared memory between the passes, so no pass ends in a barrier. Bound by the
// ranking's serial chain, below 1 us a pass against 3 us with its barriers:
// 2000 splats at 160x90 from 62.0 to 53.3 us. `p` is the first pass, keys_out
// and vals_out the sort's result.
__device__ __forceinline__ void block_sort(TileShared<8>& sm, uint32_t* s_scan, Pass p, uint32_t passes,
                                           uint32_t bits) {
  for (uint32_t pass = 0; pass < passes; ++pass) {
    uint32_t k[8], v[8], rank[8];
    rank_tile<8>(sm, s_scan, p, 0u, k, v, rank);
    arrange_tile<8>(sm, p, 0u, k, v, rank);
    p.keys_in = sm.keys;
    p.vals_in = sm.vals;
    p.shift += bits;
  }
  for (uint32_t i = threadIdx.x; i < p.n; i += kBlock) {
    p.keys_out[i] = sm.keys[i];
    p.vals_out[i] = sm.vals[i];
  }
}

// Whether a pass over n items is a tile_pass. Up to `sms` tiles of 1024 items
// (most blocks, shortest chain per block), then tiles of 2048, which keep the
// number of blocks that meet low.
__device__ __forceinline__ bool is_tile_pass(uint32_t n) { return n <= gridDim.x * kBlock * 8u; }

// A whole pass; `round` counts the sort's barriers. False: a barrier expired.
__device__ __forceinline__ bool sort_pass(FrontShared& sm, uint32_t* s_scan, const Pass& p, uint32_t* round, bool last,
                                          uint32_t small, uint32_t limit) {
  if (p.n <= small) return tile_pass<4>(sm.tile4, s_scan, p, round, last, limit);
  if (is_tile_pass(p.n)) return tile_pass<8>(sm.tile8, s_scan, p, round, last, limit);
  return chunk_pass(sm.chunk, s_scan, p, round, last, limit);
}

// Class of a tile in the raster work list, as raster.cu's.
__device__ __forceinline__ uint32_t tile_class(uint32_t samples) { return samples == 0 ? 0u : 32u - __clz(samples); }

template <bool GROUPED, bool FAST_SH, bool PERIODIC>
__global__ void __launch_bounds__(kBlock, kFrontBlocksPerSm) k_front(const __grid_constant__ Front f) {
  extern __shared__ __align__(16) unsigned char s_dyn[];
  FrontShared& sm = *reinterpret_cast<FrontShared*>(s_dyn);
  __shared__ uint32_t s_scan[kFrontWarps];
  __shared__ unsigned long long s_sum[kFrontWarps];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, c = blockIdx.x, grid = gridDim.x;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t limit = f.limit;
  uint32_t* barrier = f.frame + kFrameBarrier;
  uint32_t round = 0;
  auto expired = [&]() {
    // The rasterizer sees an overflowed frame and writes nothing, the stats
    // see the error. (The blocks that do meet at this barrier work on data
    // of earlier stages, all there; this block is missing at their next one,
    // so each of them comes here.)
    if (tid == 0) {
      atomicOr(&f.ctl->error, kErrorWait);
      atomicExch(&f.ctl->state[0], 0u);
      atomicExch(&f.ctl->state[3], 1u);
    }
  };
#define GS_MEET()                                      \
  if (!grid_barrier(barrier, ++round * grid, limit)) { \
    expired();                                         \
    return;                                            \
  }

  // Projection; block 0 clears the control block, which no one reads before
  // the first barrier.
  if (c == 0)
    for (uint32_t i = tid; i < sizeof(Control) / 4u; i += kBlock) reinterpret_cast<uint32_t*>(f.ctl)[i] = 0u;
  for (uint32_t i = c * kBlock + tid; i < 2u * front_sum_rows(grid) * kRadix; i += grid * kBlock)
    f.scratch[(size_t)grid * kRadix + i] = 0u;
  uint8_t* vis8 = reinterpret_cast<uint8_t*>(f.ordered);  // ordered is written after the depth sort
  sm.project.snorm[tid] = snorm8_value(tid);
  for (uint32_t b = c; b < f.b.total_blocks; b += grid) {
    project_block<false, GROUPED, FAST_SH, PERIODIC, true>(
        b, f.b, f.o, sm.project.snorm, sm.project.group, sm.project.count, f.mean, f.conic, f.color, f.tile_counts,
        f.keys, FAST_SH ? f.rec : nullptr, f.erec, vis8, f.frame + kFrameKeyMin, f.frame + kFrameKeyMax);
    __syncthreads();
  }
  GS_MEET();
  if (f.withhold && c == 0) return;

  // Compaction: units of 256 items, a contiguous run per block.
  const uint32_t units = f.b.total_items / kBlock;
  const uint32_t low = __ldcg(f.frame + kFrameKeyMin), high = __ldcg(f.frame + kFrameKeyMax);
  const uint32_t range = high >= low ? high - low : 0u;
  const uint32_t bits = range ? 32u - (uint32_t)__clz(range) : 0u;
  const uint32_t passes = (bits + 7u) / 8u;
  const bool odd = passes & 1u;  // start in buffer 1, so that the sorted records end up in buffer 0
  {
    const uint32_t per = (units + grid - 1u) / grid, u0 = min(c * per, units), u1 = min(u0 + per, units);
    const uint2* bytes = reinterpret_cast<const uint2*>(vis8);  // 8 warps a unit
    uint32_t before = 0, all = 0;
    const uint32_t upto = c == 0 ? units : u0;  // block 0 also counts them all
    for (uint32_t u = tid; u < upto; u += kBlock) {
      const uint2 w = bytes[u];
      const uint32_t v = __dp4a(w.x, 0x01010101u, __dp4a(w.y, 0x01010101u, 0u));
      all += v;
      before += u < u0 ? v : 0u;
    }
    before = (uint32_t)block_sum(before, s_sum);
    if (c == 0) {
      all = (uint32_t)block_sum(all, s_sum);
      if (tid < 4) f.ctl->visible_state[tid] = tid == 3 ? 0u : tid == 2 ? (all + 1023u) / 1024u : all;
    }
    for (uint32_t u = u0; u < u1; ++u) {
      const uint32_t idx = u * kBlock + tid, key = f.keys[idx];
      const bool vis = key != kInvisibleKey;
      const uint32_t bal = __ballot_sync(0xffffffffu, vis);
      const uint2 w = bytes[u];
      const unsigned long long w8 = ((unsigned long long)w.y << 32) | w.x;
      const unsigned long long below = warp ? w8 << (64u - 8u * warp) : 0ull;  // the warps before this one
      const uint32_t pos = before + __popc(bal & lt) +
                           __dp4a((uint32_t)below, 0x01010101u, __dp4a((uint32_t)(below >> 32), 0x01010101u, 0u));
      f.vis_off[idx] = pos;
      if (vis) {
        (odd ? f.dk1 : f.dk0)[pos] = key;
        (odd ? f.dv1 : f.dv0)[pos] = idx;
      }
      before += __dp4a(w.x, 0x01010101u, __dp4a(w.y, 0x01010101u, 0u));
    }
  }
  GS_MEET();

  // The depth sort's passes, then scan and emission, then the tile sort's
  // passes: one loop, so that the pass is compiled once, and in line (a call
  // keeps its arguments on the stack, in L1 lines that every barrier drops).
  const uint32_t visible = __ldcg(&f.ctl->visible_state[0]);
  const uint32_t sum_words = front_sum_rows(grid) * kRadix;
  uint32_t* sums = f.scratch + (size_t)grid * kRadix;
  uint32_t* spare = sums + sum_words;
  uint32_t count = 0;       // intersection records
  uint32_t sort_round = 0;  // barriers met within the current sort
  for (uint32_t stage = 0; stage < passes + 1u + f.tile_passes; ++stage) {
    if (stage != passes) {
      Pass p;
      if (stage < passes) {
        const bool one = odd != ((stage & 1u) != 0u);  // buffer 1 to buffer 0
        p = {one ? f.dk1 : f.dk0, one ? f.dv1 : f.dv0, one ? f.dk0 : f.dk1, one ? f.dv0 : f.dv1, visible, low,
             8u * stage, 255u, f.scratch, sums, spare, f.frame + kFrameDepthBarrier};
      } else {
        const uint32_t pass = stage - passes - 1u;
        const bool one = pass & 1u;
        p = {one ? f.tk1 : f.tk0, one ? f.tv1 : f.tv0, one ? f.tk0 : f.tk1, one ? f.tv0 : f.tv1, count, 0u,
             f.digit_bits * pass, (1u << f.digit_bits) - 1u, f.scratch, sums, spare,
             f.frame + kFrameTileBarrier};
      }
      const bool last = stage + 1u == passes || stage == passes + f.tile_passes;
      if (p.n <= kBlock * 8u) {
        const bool depth = stage < passes;
        if (c == 0) {
          p.keys_out = depth ? f.dk0 : f.tile_passes & 1u ? f.tk1 : f.tk0;
          p.vals_out = depth ? f.dv0 : f.tile_passes & 1u ? f.tv1 : f.tv0;
          block_sort(sm.tile8, s_scan, p, depth ? passes : f.tile_passes, depth ? 8u : f.digit_bits);
        }
        stage = (depth ? passes : stage + f.tile_passes) - 1u;  // all passes at once
        GS_MEET();
        continue;
      }
      if (!sort_pass(sm, s_scan, p, &sort_round, last, f.small_sort, limit)) {
        expired();
        return;
      }
      if (last) {
        GS_MEET();
        sort_round = 0;
      }
      uint32_t* used = sums;  // the spare ones are zeroed
      sums = spare;
      spare = used;
      continue;
    }
    // Tile counts in depth order and their saturating scan: runs of whole
    // warps' ranks, contiguous per block.
    const uint32_t rank_units = (visible + 31u) / 32u, rank_per = (rank_units + grid - 1u) / grid;
    const uint32_t r0 = min(c * rank_per * 32u, visible), r1 = min(r0 + rank_per * 32u, visible);
    unsigned long long sum = 0;
    for (uint32_t r = r0 + tid; r < r1; r += kBlock) {
      const uint32_t n = f.tile_counts[f.dv0[r]];
      f.ordered[r] = n;
      sum += n;
    }
    sum = block_sum(sum, s_sum);
    if (tid == 0) f.scratch[c] = (uint32_t)min(sum, 0xffffffffull);
    GS_MEET();
    unsigned long long before = 0, all = 0;
    for (uint32_t i = tid; i < grid; i += kBlock) {
      const uint32_t v = f.scratch[i];
      all += v;
      before += i < c ? v : 0u;
    }
    before = block_sum(before, s_sum);
    all = block_sum(all, s_sum);
    const uint32_t demand = (uint32_t)min(all, 0xffffffffull);  // saturating, as scan.ts:35
    const bool overflow = demand > f.capacity;
    count = overflow ? 0u : demand;
    if (c == 0 && tid == 0) {
      f.ctl->state[0] = count;
      f.ctl->state[1] = demand;
      f.ctl->state[2] = (uint32_t)(((uint64_t)count + 1023u) / 1024u);
      f.ctl->state[3] = overflow ? 1u : 0u;
      const uint32_t attempt = f.frame[kFrameAttempt];
      const uint32_t last_version = f.frame[kFrameReset] ? 0u : f.output_state[1];
      f.output_state[0] = attempt;
      f.output_state[1] = overflow ? last_version : attempt;
      f.output_state[2] = demand;
      f.output_state[3] = overflow ? 1u : 0u;
    }
    // Offsets and emission, 256 ranks at a time.
    for (uint32_t r = r0; r < r1; r += kBlock) {
      const uint32_t mine = r + tid;
      const bool live = mine < r1;
      const uint32_t g = live ? f.dv0[mine] : 0u, reserved = live ? f.ordered[mine] : 0u;
      uint32_t total;
      const uint32_t excl = block_exclusive_scan<true>(reserved, s_scan, &total);
      const uint32_t offset = (uint32_t)min(before + excl, 0xffffffffull);
      if (live) f.ioff[mine] = offset;
      before += total;
      if (!overflow) {
        float4 e0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), e1 = e0;
        if (live) {
          e0 = f.erec[2 * (size_t)g];
          e1 = f.erec[2 * (size_t)g + 1];
        }
        emit_group<PERIODIC>(sm.emit, live, g, e0, e1, reserved, offset, f.b, f.o, f.capacity, f.tk0, f.tv0);
      }
    }
    GS_MEET();
  }

  // Tile ranges: offsets[t] = first sorted index with tile >= t.
  const uint32_t* sorted = f.tile_passes & 1u ? f.tk1 : f.tk0;
  const uint32_t ntile = f.b.total_tiles;
  for (uint64_t i = (uint64_t)c * kBlock + tid; i <= count; i += (uint64_t)grid * kBlock) {
    const uint32_t lo = i == 0 ? 0u : sorted[i - 1] + 1u, hi = i == count ? ntile : min(sorted[i], ntile);
    for (uint32_t t = lo; t <= hi; ++t) f.tile_offsets[t] = (uint32_t)i;
  }
  if (!f.tile_order) return;
  GS_MEET();

  // Raster work list, heaviest class first (raster.cu: k_order_count, k_order_scatter).
  uint32_t* s_class = reinterpret_cast<uint32_t*>(s_dyn);  // counts, then bases, of the 34 classes
  uint32_t* s_start = s_class + 64;
  for (uint32_t t0 = c * kBlock; t0 < ntile; t0 += grid * kBlock) {
    if (tid < 34u) s_class[tid] = 0u;
    __syncthreads();
    const uint32_t t = t0 + tid;
    if (t < ntile) atomicAdd(&s_class[tile_class(f.tile_offsets[t + 1] - f.tile_offsets[t])], 1u);
    __syncthreads();
    if (tid < 34u && s_class[tid]) atomicAdd(&f.ctl->order_hist[tid], s_class[tid]);
    __syncthreads();
  }
  GS_MEET();
  if (tid == 0) {
    uint32_t run = 0;
    for (int k = 33; k >= 0; --k) {
      s_start[k] = run;
      run += __ldcg(&f.ctl->order_hist[k]);
    }
  }
  for (uint32_t t0 = c * kBlock; t0 < ntile; t0 += grid * kBlock) {
    __syncthreads();
    if (tid < 34u) s_class[tid] = 0u;
    __syncthreads();
    const uint32_t t = t0 + tid;
    uint32_t k = 0, local = 0;
    if (t < ntile) {
      k = tile_class(f.tile_offsets[t + 1] - f.tile_offsets[t]);
      local = atomicAdd(&s_class[k], 1u);
    }
    __syncthreads();
    if (tid < 34u && s_class[tid]) s_class[tid] = atomicAdd(&f.ctl->order_fill[tid], s_class[tid]);
    __syncthreads();
    if (t < ntile) f.tile_order[s_start[k] + s_class[k] + local] = t;
  }
#undef GS_MEET
}

const void* front_kernel(bool grouped, bool fast, bool periodic) {
  if (grouped) {
    if (fast) return periodic ? (const void*)k_front<true, true, true> : (const void*)k_front<true, true, false>;
    return periodic ? (const void*)k_front<true, false, true> : (const void*)k_front<true, false, false>;
  }
  if (fast) return periodic ? (const void*)k_front<false, true, true> : (const void*)k_front<false, true, false>;
  return periodic ? (const void*)k_front<false, false, true> : (const void*)k_front<false, false, false>;
}

}  // namespace

size_t front_scratch_words(int sms) {
  const uint32_t grid = kFrontBlocksPerSm * (uint32_t)sms;
  return (size_t)(grid + 2u * front_sum_rows(grid)) * kRadix;
}

static_assert(sizeof(FrontShared) <= 48 * 1024, "a larger size has to be opted into");

bool front_fits(int device) {
  // Asked once per device (the answers do not change): 0 not yet, 1 no, 2 yes.
  static std::atomic<int> known[64];
  const bool keep = device >= 0 && device < 64;
  if (keep && known[device].load()) return known[device].load() == 2;
  int cooperative = 0;
  bool ok = cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, device) == cudaSuccess && cooperative;
  for (int i = 0; i < 8; ++i) {
    int blocks = 0;
    ok = ok && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, front_kernel(i & 1, i & 2, i & 4), kBlock,
                                                             sizeof(FrontShared)) == cudaSuccess &&
         blocks >= (int)kFrontBlocksPerSm;
  }
  if (!ok) cudaGetLastError();
  if (keep) known[device].store(ok ? 2 : 1);
  return ok;
}

cudaError_t launch_front(const BatchView& b, const PassOptions& o, const FrontBuffers& w, uint32_t* frame_params,
                         uint32_t capacity, uint32_t tile_passes, uint32_t digit_bits, int sms, uint32_t wait_limit,
                         bool withhold, cudaStream_t st) {
  Front f;
  f.b = b;
  f.o = o;
  f.mean = w.mean; f.conic = w.conic; f.color = w.color; f.rec = w.rec; f.erec = w.erec;
  f.tile_counts = w.tile_counts; f.keys = w.keys; f.vis_off = w.vis_off;
  f.ordered = w.ordered; f.ioff = w.ioff;
  f.dk0 = w.dk[0]; f.dk1 = w.dk[1]; f.dv0 = w.dv[0]; f.dv1 = w.dv[1];
  f.tk0 = w.tk[0]; f.tk1 = w.tk[1]; f.tv0 = w.tv[0]; f.tv1 = w.tv[1];
  f.tile_offsets = w.tile_offsets; f.tile_order = w.tile_order;
  f.scratch = w.scratch;
  f.ctl = w.ctl;
  f.frame = frame_params;
  f.output_state = w.output_state;
  f.capacity = capacity;
  f.tile_passes = tile_passes;
  f.digit_bits = digit_bits;
  f.limit = wait_limit ? wait_limit : kSpinLimit;
  f.withhold = withhold ? 1u : 0u;
  // A block per 256 ordinals (the views of a group share projection blocks, but
  // no later stage), at least one and at most kFrontBlocksPerSm per SM (all of
  // them resident: the blocks wait on one another).
  const uint32_t grid = std::min(std::max(b.total_items / kBlock, (uint32_t)sms), kFrontBlocksPerSm * (uint32_t)sms);
  f.small_sort = std::min(grid, (uint32_t)sms) * kBlock * 4u;
  void* args[] = {&f};
  return cudaLaunchCooperativeKernel(front_kernel(b.ngroups < b.nviews, w.rec != nullptr, o.axis != 0u), dim3(grid),
                                     dim3(kBlock), args, sizeof(FrontShared), st);
}

}  // namespace gs
