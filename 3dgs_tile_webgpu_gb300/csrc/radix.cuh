// One chunk of a stable LSD radix sort pass: digit counts of its keys, and the
// scatter of a tile (sort.cu has the whole pass, and what bounds it).
// Shared by the sort kernels (sort.cu) and the fused front of small launches
// (front.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "pass_common.cuh"

namespace gs {

constexpr int kCountWarps = kBlock / 32;
constexpr int kScatterThreads = 256;
constexpr int kSortWarps = kScatterThreads / 32;

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

// Tiles [t0, t1), of `tile` items each, of chunk c when n items split over `chunks` chunks.
__device__ __forceinline__ void chunk_tiles(uint32_t n, uint32_t tile, uint32_t chunks, uint32_t c, uint32_t* t0,
                                            uint32_t* t1) {
  const uint32_t tiles = (uint32_t)(((uint64_t)n + tile - 1) / tile);
  *t0 = (uint32_t)((uint64_t)c * tiles / chunks);
  *t1 = (uint32_t)((uint64_t)(c + 1u) * tiles / chunks);
}

// Adds the digits of keys [begin, end) to the warps' rows of hist, called by a
// whole block of kBlock threads; begin is a multiple of 4.
template <int BITS, class Digit>
__device__ __forceinline__ void count_keys(uint32_t (*hist)[1u << BITS], const uint32_t* keys, uint32_t begin,
                                           uint32_t end, const Digit& digit) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  // Each warp takes 512-key runs: four 16-byte loads per lane in flight
  // before any counting (begin is a multiple of 4, so they are aligned).
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
      const uint32_t d = digit(kk[q]);
      const uint32_t d0 = __shfl_sync(0xffffffffu, d, 0);
      if (__all_sync(0xffffffffu, ok && d == d0)) {
        if (lane == 0u) atomicAdd(&hist[warp][d0], 32u);
      } else if (ok) {
        atomicAdd(&hist[warp][d], 1u);
      }
    }
  }
}

// Digits owned by a thread of the scatter.
__host__ __device__ constexpr int digits_per_thread(int bits) { return bits > 8 ? 2 : 1; }

template <int BITS>
struct ScatterShared {
  uint16_t warp_hist[kSortWarps][1u << BITS];  // a warp's items per digit, then its first tile position
  uint32_t match[kSortWarps][1u << BITS];  // lanes of the warp's current row holding each digit; zero in between
  uint32_t delta[1u << BITS];  // global position of the tile's item i of a digit, minus i
  uint32_t scan[8];
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

// Ranks the tile of kScatterThreads * ITEMS items held in kb/vb (items from base
// on, those below n),
// stages it in place in block-sorted order and writes each digit's run to its
// global position. FULL: every item of the tile is below n. `run`: the global
// position of the next item of digit threadIdx.x (threads below 2^BITS).
// Leaves warp_hist zeroed and run advanced past the tile. landed(): waits until
// the warp's own values (32 * ITEMS from wofs on) are in vb; false if they never
// came, and then of scatter_tile.
template <int BITS, int ITEMS, bool FULL, class Digit, class Landed>
__device__ __forceinline__ bool scatter_tile(ScatterShared<BITS>& sm, uint32_t* kb, uint32_t* vb, uint32_t base,
                                             uint32_t n, const Digit& digit, uint32_t* keys_out, uint32_t* vals_out,
                                             uint32_t (&run)[digits_per_thread(BITS)], const Landed& landed) {
  constexpr uint32_t RADIX = 1u << BITS;
  constexpr int D = digits_per_thread(BITS);
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t wofs = warp * 32u * ITEMS;  // warp-striped: item j*32+lane of the warp's segment
  uint32_t k[ITEMS], rank[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) k[j] = kb[wofs + (uint32_t)j * 32u + lane];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const bool ok = FULL || base + wofs + (uint32_t)j * 32u + lane < n;
    const uint32_t valid = FULL ? 0xffffffffu : __ballot_sync(0xffffffffu, ok);
    const uint32_t d = digit(k[j]);
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
  for (int j = 0; j < ITEMS; ++j) {
    if (FULL || base + wofs + (uint32_t)j * 32u + lane < n) {
      const uint32_t d = digit(k[j]);
      rank[j] += sm.warp_hist[warp][d];
      kb[rank[j]] = k[j];
    }
  }
  const bool there = landed();
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) k[j] = vb[wofs + (uint32_t)j * 32u + lane];
  if (!__syncthreads_and(there)) return false;
#pragma unroll
  for (int j = 0; j < ITEMS; ++j)
    if (FULL || base + wofs + (uint32_t)j * 32u + lane < n) vb[rank[j]] = k[j];
  __syncthreads();

  constexpr uint32_t kTile = kScatterThreads * ITEMS;
  const uint32_t items = FULL ? kTile : min(kTile, n - base);
#pragma unroll 4
  for (uint32_t i = tid; i < items; i += kScatterThreads) {
    const uint32_t key = kb[i];
    const uint32_t dst = sm.delta[digit(key)] + i;
    keys_out[dst] = key;
    vals_out[dst] = vb[i];
  }
  for (uint32_t i = tid; i < kSortWarps * RADIX * sizeof(uint16_t) / 4u; i += kScatterThreads)
    reinterpret_cast<uint32_t*>(&sm.warp_hist[0][0])[i] = 0u;
  __syncthreads();
  return true;
}

}  // namespace gs
