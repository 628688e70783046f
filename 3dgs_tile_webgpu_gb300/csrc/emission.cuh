// Emission of one group of depth ranks, shared by the emission kernel
// (pass_exact.cu) and the fused front of small launches (front.cu). Only
// compiled in translation units built with --fmad=false.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "pass_common.cuh"
#include "projection.cuh"

namespace gs {

// ---------------------------------------------------------------------------
// Intersection emission (intersections.ts:43-111): per depth rank, one
// (tile, item) record for every tile the splat contributes to, written at the
// rank's scanned offset; sentinel padding if fewer hits than reserved. Tile
// ids are global over the batch (the view's tile_base + local id; the
// sentinel is the batch's tile total).
//
// Warp-cooperative: a warp owns 32 consecutive depth ranks and spreads the
// union of their bounding-box tiles over its lanes, 32 box tiles per round,
// so one wide splat no longer idles the other 31 lanes. Each lane finds the
// rank owning its box tile by a binary search over the warp's inclusive box
// counts, runs the reference's tile test, and places a hit after the owner's
// earlier hits (owner's running count + hits of lower lanes with the same
// owner this round). A splat's records thus fill its reserved range in
// row-major box order, the order of the per-splat loop; the record set per
// splat is what the stable tile sort sees, so the sorted result is the same.
// Boxes of kRowBox tiles or more take rounds of 32 box rows instead: a lane
// finds the run of tiles its row emits (row_span, as the projection's count
// did), and the warp's lanes write the runs, one record each.
constexpr int kEmitWarps = kBlock / 32;

struct EmitShared {
  float f[10][kEmitWarps][32];     // cx, cy, conic a, b, c, threshold, rx, ry, view width, height
  uint32_t u[10][kEmitWarps][32];  // box x0, y0, width, tiles_x, tile_base, base, reserved, item,
                                   // first box tile of the warp's walk, wrap
  uint32_t own[kEmitWarps][32];    // lane owning the k-th segment of the round; box rows: their records, inclusive
  uint32_t filled[kEmitWarps][32]; // records placed so far per rank
};

// Emits the boxes of the lanes with rows != 0 (their heights) in rounds of 32
// box rows, the boxes end to end in lane order; sm.filled counts the records.
// (Not inlining this and emit_wide: 82 us instead of 76 for 2.3M ranks.)
__device__ __forceinline__ void emit_rows(EmitShared& sm, uint32_t rows, float ts, float inv, uint32_t capacity,
                                              uint32_t* __restrict__ tile_keys, uint32_t* __restrict__ tile_vals) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  sm.u[8][warp][lane] = warp_inclusive(rows);
  __syncwarp();
  const uint32_t total = sm.u[8][warp][31];
  for (uint32_t j0 = 0; j0 < total; j0 += 32) {
    const uint32_t j = j0 + lane;
    const bool valid = j < total;
    uint32_t owner = 0, row = 0, n = 0, height = 0;
    int first = 0, ty = 0;
    if (valid) {
      owner = find_owner(sm.u[8][warp], j);
      const uint32_t start = owner ? sm.u[8][warp][owner - 1] : 0u;
      row = j - start;
      height = sm.u[8][warp][owner] - start;
      first = (int)sm.u[0][warp][owner];
      ty = (int)(sm.u[1][warp][owner] + row);
      n = sm.u[2][warp][owner];
      if (sm.u[6][warp][owner] != n * height) {  // not every box tile passed
        const RowSpan r = row_span(sm.f[0][warp][owner], sm.f[1][warp][owner], sm.f[2][warp][owner],
                                   sm.f[3][warp][owner], sm.f[4][warp][owner], sm.f[5][warp][owner], ty, first,
                                   first + (int)n - 1, sm.f[8][warp][owner] + sm.f[9][warp][owner], ts,
                                   inv);
        first = r.first;
        n = r.last >= r.first ? (uint32_t)(r.last - r.first + 1) : 0u;
      }
    }
    // The row's records follow those of the owner's earlier rows: past
    // rounds' (filled), then the lanes' below it from the owner's first on.
    const uint32_t incl = warp_inclusive(n);
    const uint32_t before = __shfl_sync(0xffffffffu, incl - n, valid && row <= lane ? lane - row : 0u);
    // The row's first record's place, the end of the rank's range, the first
    // tile and the item, handed to the writing lanes by shuffles.
    uint32_t place = 0, end = 0, tile = 0, item = 0;
    if (valid) {
      const uint32_t base = sm.u[5][warp][owner];
      place = base + sm.filled[warp][owner] + (incl - n - before);
      end = min(base + sm.u[6][warp][owner], capacity);
      tile = sm.u[4][warp][owner] + (uint32_t)ty * sm.u[3][warp][owner] + (uint32_t)first;
      item = sm.u[7][warp][owner];
    }
    sm.own[warp][lane] = incl;
    __syncwarp();
    if (valid && (row + 1u == height || lane == 31u)) sm.filled[warp][owner] = place + n - sm.u[5][warp][owner];
    const uint32_t records = sm.own[warp][31];
    for (uint32_t q0 = 0; q0 < records; q0 += 32) {
      const uint32_t q = q0 + lane, l = find_owner(sm.own[warp], min(q, records - 1u));
      const uint32_t off = q - (l ? sm.own[warp][l - 1] : 0u);
      const uint32_t dst = __shfl_sync(0xffffffffu, place, l) + off;
      const uint32_t stop = __shfl_sync(0xffffffffu, end, l);
      const uint32_t key = __shfl_sync(0xffffffffu, tile, l) + off;
      const uint32_t val = __shfl_sync(0xffffffffu, item, l);
      if (q < records && dst < stop) {
        tile_keys[dst] = key;
        tile_vals[dst] = val;
      }
    }
    __syncwarp();  // the tables are rewritten by the next round
  }
}

// The boxes of the lanes in `lanes` (nbox tiles each), emitted one at a time by
// the whole warp, 32 tiles a step in row-major box order, each hit after the
// box's earlier hits; returns each of these lanes' record count.
template <bool PERIODIC>
__device__ __forceinline__ uint32_t emit_wide(EmitShared& sm, uint32_t lanes, uint32_t nbox, uint32_t axis,
                                                  float ts, uint32_t capacity, uint32_t* __restrict__ tile_keys,
                                                  uint32_t* __restrict__ tile_vals) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  // The owner's parameters are read from the warp's table at each step
  // (broadcast loads) rather than held in registers across the walk.
  const volatile float(*vf)[kEmitWarps][32] = sm.f;
  const volatile uint32_t(*vu)[kEmitWarps][32] = sm.u;
  uint32_t filled = 0;
  while (lanes) {
    const uint32_t w = (uint32_t)__ffs(lanes) - 1u;
    lanes &= lanes - 1u;
    const uint32_t wn = __shfl_sync(0xffffffffu, nbox, w);
    const uint32_t wres = vu[6][warp][w];
    const bool wfull = wres == wn;
    uint32_t wfilled = 0;
    for (uint32_t k0 = 0; k0 < wn; k0 += 32) {
      const uint32_t k = k0 + lane;
      bool hit = false;
      uint32_t t = 0;
      if (k < wn) {
        const uint32_t wbw = vu[2][warp][w];
        const uint32_t by = k / wbw, bx = k - by * wbw;
        const int tx = box_column<PERIODIC>(bx, vu[0][warp][w], vu[9][warp][w], axis);
        const int ty = box_row<PERIODIC>(by, vu[1][warp][w], vu[9][warp][w], axis);
        hit = wfull || tile_hit<PERIODIC>(vf[0][warp][w], vf[1][warp][w], vf[2][warp][w], vf[3][warp][w],
                                          vf[4][warp][w], vf[5][warp][w], vf[6][warp][w], vf[7][warp][w], tx,
                                          ty, vf[8][warp][w], vf[9][warp][w], axis, ts);
        t = vu[4][warp][w] + (uint32_t)ty * vu[3][warp][w] + (uint32_t)tx;
      }
      const uint32_t hits = __ballot_sync(0xffffffffu, hit);
      if (hit) {
        const uint32_t local = wfilled + __popc(hits & lt);
        const uint32_t wbase = vu[5][warp][w];
        if (local < wres && wbase + local < capacity) {
          tile_keys[wbase + local] = t;
          tile_vals[wbase + local] = vu[7][warp][w];
        }
      }
      wfilled += __popc(hits);
    }
    if (lane == w) filled = wfilled;
  }
  return filled;
}

// One group of kBlock depth ranks (32 per warp): stage each lane's box and
// tile-test inputs for its warp, walk the union of the warp's boxes 32 box
// tiles per round, place hits after the owner's earlier hits, pad with
// sentinels. The lane's rank data were loaded by the caller.
template <bool PERIODIC>
__device__ __forceinline__ void emit_group(EmitShared& sm, bool live, uint32_t g, float4 e0, float4 e1,
                                           uint32_t reserved, uint32_t base_off, const BatchView& bv,
                                           const PassOptions& o, uint32_t capacity, uint32_t* __restrict__ tile_keys,
                                           uint32_t* __restrict__ tile_vals) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t sentinel = bv.total_tiles;
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t nbox = 0, rows = 0;
  if (live) {
    const ViewDesc& v = bv.views[find_view(bv.item_base, bv.nviews, g)];
    // Emission record: (cx, cy, conic a, b), (conic c, threshold, rx + 512 ry, tile walk).
    const float4 m = make_float4(e0.x, e0.y, 0.0f, 0.0f), c = make_float4(e0.z, e0.w, e1.x, 0.0f);
    const uint32_t packed = (uint32_t)e1.z;
    const float rx = (float)(packed % 512u), ry = (float)(packed / 512u);
    const float thr = e1.y;  // log(opacity * 255), computed by the projection
    const TileBox box = tile_box<PERIODIC>(m.x, m.y, rx, ry, v.vw, v.vh, (int)v.tiles_x, (int)v.tiles_y, o);
    // A rank with nothing reserved emits nothing; its box takes no rounds.
    nbox = reserved ? box.bw * box.bh : 0u;
    rows = box.bh;
    sm.f[0][warp][lane] = m.x; sm.f[1][warp][lane] = m.y;
    sm.f[2][warp][lane] = c.x; sm.f[3][warp][lane] = c.y; sm.f[4][warp][lane] = c.z;
    sm.f[5][warp][lane] = thr; sm.f[6][warp][lane] = rx; sm.f[7][warp][lane] = ry;
    sm.f[8][warp][lane] = v.vw; sm.f[9][warp][lane] = v.vh;
    sm.u[0][warp][lane] = (uint32_t)box.x0; sm.u[1][warp][lane] = (uint32_t)box.y0; sm.u[2][warp][lane] = box.bw;
    sm.u[3][warp][lane] = v.tiles_x; sm.u[4][warp][lane] = v.tile_base;
    if (PERIODIC) sm.u[9][warp][lane] = box.wrap;
    sm.u[5][warp][lane] = base_off; sm.u[6][warp][lane] = reserved; sm.u[7][warp][lane] = g;
  }
  const uint32_t le = lt | (1u << lane);
  sm.filled[warp][lane] = 0u;
  uint32_t filled = 0;
  // A splat whose every box tile passed the projection's count (reserved ==
  // nbox) emits its whole box: those boxes are walked first without the tile
  // test, the others after it with the test. Each splat is walked once, so
  // its records keep row-major box order. The boxes the projection counted by
  // rows follow, then those it walked one at a time (count_tiles_warp).
  const bool full = reserved == nbox;
  const bool by_rows = !PERIODIC && nbox >= kRowBox && e1.w == 0.0f;
  const bool wide = PERIODIC ? nbox >= kWideBox : nbox >= kRowBox && !by_rows;
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    const uint32_t nb = !wide && !by_rows && (pass == 0) == full ? nbox : 0u;
    uint32_t incl = nb;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= (uint32_t)d) incl += y;
    }
    const uint32_t excl = incl - nb;
    sm.u[8][warp][lane] = excl;
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);

    // Rounds of 32 box tiles. The boxes lie end to end in lane order, so a
    // round is a run of segments, one per owning lane: a lane finds its
    // segment from the OR of the segment starts and the segment's owner from
    // a table the owners wrote; each owner adds its hits under its own mask.
    for (uint32_t j0 = 0; j0 < total; j0 += 32) {
      const uint32_t lo = max(excl, j0), hi = min(incl, j0 + 32u);
      const bool seg = lo < hi;
      const uint32_t starts = __reduce_or_sync(0xffffffffu, seg ? 1u << (lo - j0) : 0u);
      const uint32_t owners = __ballot_sync(0xffffffffu, seg);
      if (seg) sm.own[warp][__popc(owners & lt)] = lane;
      __syncwarp();
      const uint32_t j = j0 + lane;
      const bool valid = j < total;
      uint32_t owner = 0, seg_start = 0;
      bool hit = false;
      uint32_t t = 0;
      if (valid) {
        const uint32_t mine = starts & le;
        owner = sm.own[warp][__popc(mine) - 1u];
        seg_start = 31u - (uint32_t)__clz(mine);
        const uint32_t bw = sm.u[2][warp][owner];
        const uint32_t kk = j - sm.u[8][warp][owner];
        const uint32_t by = kk / bw, bx = kk - by * bw;
        const int tx = box_column<PERIODIC>(bx, sm.u[0][warp][owner], sm.u[9][warp][owner], o.axis);
        const int ty = box_row<PERIODIC>(by, sm.u[1][warp][owner], sm.u[9][warp][owner], o.axis);
        hit = pass == 0 ||
              tile_hit<PERIODIC>(sm.f[0][warp][owner], sm.f[1][warp][owner], sm.f[2][warp][owner],
                                sm.f[3][warp][owner], sm.f[4][warp][owner], sm.f[5][warp][owner],
                                sm.f[6][warp][owner], sm.f[7][warp][owner], tx, ty, sm.f[8][warp][owner],
                                sm.f[9][warp][owner], o.axis, o.tile_px);
        t = sm.u[4][warp][owner] + (uint32_t)ty * sm.u[3][warp][owner] + (uint32_t)tx;
      }
      const uint32_t hits = __ballot_sync(0xffffffffu, hit);
      if (hit) {
        // After the owner's earlier hits: those of past rounds, then those of
        // this round below this lane within the owner's segment.
        const uint32_t local = sm.filled[warp][owner] + __popc(hits & lt & ~((1u << seg_start) - 1u));
        const uint32_t base = sm.u[5][warp][owner];
        if (local < sm.u[6][warp][owner] && base + local < capacity) {
          tile_keys[base + local] = t;
          tile_vals[base + local] = sm.u[7][warp][owner];
        }
      }
      __syncwarp();  // every read of filled, the owner table and the walk bases is done
      if (seg) {
        filled += __popc(hits & bit_range(lo - j0, hi - j0));
        sm.filled[warp][lane] = filled;
      }
    }
    __syncwarp();
  }

  if (!PERIODIC && __any_sync(0xffffffffu, by_rows)) {
    emit_rows(sm, by_rows ? rows : 0u, o.tile_px, o.tile_inv, capacity, tile_keys, tile_vals);
    if (by_rows) filled = sm.filled[warp][lane];
  }

  const uint32_t wide_lanes = __ballot_sync(0xffffffffu, wide);
  if (wide_lanes) {
    const uint32_t n = emit_wide<PERIODIC>(sm, wide_lanes, nbox, o.axis, o.tile_px, capacity, tile_keys, tile_vals);
    if (wide) filled = n;
  }

  // Sentinel padding for reserved slots without a hit.
  if (live) {
    for (uint32_t pad = filled; pad < reserved; ++pad)
      if (base_off + pad < capacity) {
        tile_keys[base_off + pad] = sentinel;
        tile_vals[base_off + pad] = g;
      }
  }
  __syncwarp();  // the warp's tables are rewritten by the next group
}

}  // namespace gs
