// Projection of one block of ordinals, shared by the projection kernel
// (pass_exact.cu) and the fused front of small launches (front.cu). Only
// compiled in translation units built with --fmad=false.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "pass_common.cuh"
#include "raster_impl.cuh"
#include "splat_math.cuh"

namespace gs {

// ---------------------------------------------------------------------------
// K1: decode + project + cull + SH + tile count, one thread per active ordinal
// of every view group (ProjectionStage.ts:385-649): consecutive views of a
// batch that render the same packed scene form a group, and each thread
// decodes its splat once and projects it into every view of the group. Writes
// the projected mean/conic/colour/count like the reference, plus the depth
// sort key (or kInvisibleKey), which the compaction consumes instead of
// re-reading the 16-byte means. Each block belongs to one group; the padding
// items after a view's last ordinal are written as invisible.
__device__ __forceinline__ void load_sh(const uint32_t* __restrict__ p, uint32_t degree, uint32_t* co) {
  if (degree == 3) {
    const uint4* v = reinterpret_cast<const uint4*>(p);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint4 w = __ldg(v + i);
      co[4 * i] = w.x; co[4 * i + 1] = w.y; co[4 * i + 2] = w.z; co[4 * i + 3] = w.w;
    }
  } else {
    // Fully unrolled with constant indices so co[] stays in registers.
    const uint32_t C = (degree + 1) * (degree + 1);
#pragma unroll
    for (uint32_t i = 0; i < 16; ++i) co[i] = i < C ? __ldg(p + i) : 0u;
  }
}

// FAST: the colour feeds only a fast raster form (eval_sh_fast); otherwise
// the reference's expression order (eval_sh, bit-exact with the oracle).
template <bool FAST>
__device__ __forceinline__ f3 eval_sh_any(uint32_t degree, const uint32_t* co, f3 d, const float* snorm) {
  if (FAST) {
    switch (degree) {
      case 0: return eval_sh_fast<0>(co, d);
      case 1: return eval_sh_fast<1>(co, d);
      case 2: return eval_sh_fast<2>(co, d);
      default: return eval_sh_fast<3>(co, d);
    }
  }
  switch (degree) {
    case 0: return eval_sh<0>(co, d, snorm);
    case 1: return eval_sh<1>(co, d, snorm);
    case 2: return eval_sh<2>(co, d, snorm);
    default: return eval_sh<3>(co, d, snorm);
  }
}

// Bits [s, e) of a word, 0 <= s < e <= 32.
__device__ __forceinline__ uint32_t bit_range(uint32_t s, uint32_t e) {
  return (e >= 32u ? 0xffffffffu : ((1u << e) - 1u)) & ~((1u << s) - 1u);
}

// Boxes along a periodic axis of at least this many tiles are walked by the
// whole warp, one box at a time, instead of in the shared rounds of the tile
// count and the emission: no per-tile owner lookup, the owner's parameters
// broadcast to every lane.
constexpr uint32_t kWideBox = 64;

// The tiles a splat may reach, walked in row-major order: bw columns and bh
// rows. Along a periodic axis the reference takes every tile of the axis and
// tests each (projectionHelpers.ts:223-236); the box keeps those that an
// image of the splat's extent can touch, which is one interval or, across the
// seam, a first part [0, wrap) and a last part from x0 + wrap (y0 + wrap) on.
struct TileBox {
  int x0, y0;
  uint32_t bw, bh;
  uint32_t wrap;  // periodic axis: box columns (rows) of the first part

};

// The tile test of box column bx and row by. PERIODIC: o.axis is not 0 (the
// kernels are compiled for both, so that plain boxes carry no axis tests and
// no wrap: sharing the code cost the projection 1%).
template <bool PERIODIC>
__device__ __forceinline__ int box_column(uint32_t bx, uint32_t x0, uint32_t wrap, uint32_t axis) {
  return (int)(PERIODIC && axis == 1u && bx < wrap ? bx : x0 + bx);
}
template <bool PERIODIC>
__device__ __forceinline__ int box_row(uint32_t by, uint32_t y0, uint32_t wrap, uint32_t axis) {
  return (int)(PERIODIC && axis == 2u && by < wrap ? by : y0 + by);
}
template <bool PERIODIC>
__device__ __forceinline__ bool tile_hit(float cx, float cy, float k0, float k1, float k2, float thr, float rx,
                                         float ry, int tx, int ty, float vw, float vh, uint32_t axis, float ts) {
  return PERIODIC ? boundary_tile_hit(cx, cy, k0, k1, k2, thr, rx, ry, tx, ty, vw, vh, axis, ts)
                  : tile_rect_test(cx, cy, k0, k1, k2, thr, tx, ty, ts);
}

// The tiles of a periodic axis that pass boundary_tile_hit's image range
// (tileContribution.ts:84-114) for some image, or more: an image centre
// canon + i period reaches tile t when it lies in [t ts - r, (t + 1) ts + r].
// The slack of 2 px and a millionth of the period covers the rounding of that
// range. Every image but i = -1, 0, 1 is out of reach, and at most one of
// i = -1 and i = 1 in it, when the extent stays well below half the period;
// otherwise (or with a centre so far out that canon is not in the period)
// the whole axis is kept. Walking 128 columns for the 2-3 that can hit took
// 367 us in the projection and 391 us in the emission of 400k splats at
// 2048x1024 (of 1384 us for the frame); 45 and 23 us so.
__device__ __forceinline__ void periodic_tiles(float cen, float r, float period, int tiles, float ts, float inv,
                                               int* start, uint32_t* count, uint32_t* wrap) {
  *start = 0; *count = (uint32_t)tiles; *wrap = 0u;
  const float canon = cen - floorf(cen / period) * period;
  const float reach = r + 2.0f + 1e-6f * period;
  if (!(canon >= 0.0f && canon <= period && 2.0f * (reach + ts) < period)) return;
  const int last = tiles - 1;
  const int a = max((int)floorf((canon - reach) * inv), 0), b = min((int)floorf((canon + reach) * inv), last);
  const float before = canon - period + reach, after = canon + period - reach;
  if (before >= 0.0f) {  // image -1 reaches the first tiles, image 0 the last one
    const int n0 = (int)floorf(before * inv) + 1;
    *wrap = (uint32_t)n0; *start = a - n0; *count = (uint32_t)(n0 + tiles - a);
  } else if (after <= (float)tiles * ts) {  // image 1 reaches the last tiles, image 0 the first one
    const int f = min((int)floorf(after * inv), last), n0 = b + 1;
    *wrap = (uint32_t)n0; *start = f - n0; *count = (uint32_t)(n0 + tiles - f);
  } else {
    *start = a; *count = (uint32_t)(b - a + 1);
  }
}

template <bool PERIODIC>
__device__ __forceinline__ TileBox tile_box(float cx, float cy, float rx, float ry, float vw, float vh, int tiles_x,
                                            int tiles_y, const PassOptions& o) {
  const float mtx = (float)(tiles_x - 1), mty = (float)(tiles_y - 1);
  // Division by the tile side, a power of two: the product with its
  // reciprocal is the same correctly rounded value.
  const int tminx = (int)clampf(floorf((cx - rx) * o.tile_inv), 0.0f, mtx);
  const int tminy = (int)clampf(floorf((cy - ry) * o.tile_inv), 0.0f, mty);
  const int tmaxx = (int)clampf(floorf((cx + rx) * o.tile_inv), 0.0f, mtx);
  const int tmaxy = (int)clampf(floorf((cy + ry) * o.tile_inv), 0.0f, mty);
  TileBox t = {tminx, tminy, (uint32_t)(tmaxx - tminx + 1), (uint32_t)(tmaxy - tminy + 1), 0u};
  if (PERIODIC && o.axis == 1u) periodic_tiles(cx, rx, vw, tiles_x, o.tile_px, o.tile_inv, &t.x0, &t.bw, &t.wrap);
  if (PERIODIC && o.axis == 2u) periodic_tiles(cy, ry, vh, tiles_y, o.tile_px, o.tile_inv, &t.y0, &t.bh, &t.wrap);
  return t;
}

// Boxes of at least this many tiles are counted and emitted row by row
// (row_span): a lane finds the tiles of one box row that pass the reference's
// tile test without testing each. Projection and emission, us, with all boxes
// walked tile by tile and with rows from 96 / 64 / 32 / 12 tiles on: 12M
// splats at 4K (398M records) 4074 + 3767, and 2814 + 2344, 2668 + 2245,
// 2486 + 2105, 2384 + 1948; 16 views of 3M splats (85M records, mostly small
// boxes) 2877 + 1106, and 2849 + 1198, 2849 + 1198, 2863 + 1202, 3236 + 1270
// (an emission kernel since replaced: 1737 and 1098 from 32 on).
constexpr uint32_t kRowBox = 32;

__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The tiles of one box row that pass tile_rect_test, [first, last] (empty:
// last < first). Not `regular`: the row's hits are not one run, or the conic is
// too near singular to bound the test's rounding; the box is then walked tile
// by tile.
struct RowSpan {
  int first, last;
  bool regular;
};

// The splat's support {q(d) <= 2 thr}, cut by the row's y range, projects onto an
// interval of x; a tile passes when it meets the interval. The ends follow
// from the conic: the support's rightmost point lies at dy = -(k1 / k2) X with
// X = sqrt(2 thr k2 / det), its boundary at dy is
// x = (-k1 dy +- sqrt(2 thr k0 - det dy^2)) / k0, and the end over the row is
// the boundary at that dy clamped to the row. The interval is taken once with
// the threshold raised by `delta` and the row and the ends widened by `m`
// pixels, once with both the other way: tiles outside the wide one fail, tiles
// that meet the narrow one pass, and those between (mostly none) are tested as
// the reference does. delta and m bound the rounding of the reference's test:
// its sigma is off by at most a few 2^-24 times k0 dx^2 + k2 dy^2 + 2 |k1 dx dy|,
// which at the boundary is below 4 k0 k2 / det thr, and its dx, dy by a
// few units in the last place of the coordinates.
__device__ __forceinline__ RowSpan row_span(float cx, float cy, float k0, float k1, float k2, float thr, int ty,
                                            int x0, int x1, float extent, float ts, float inv) {
  RowSpan s = {1, 0, true};
  const float p = k1 * k1;
  const float det = __fmaf_rn(k0, k2, -p) - __fmaf_rn(k1, k1, -p);  // k0 k2 - k1^2 without its cancellation error
  const float delta = 1e-3f + 4e-6f * __fdividef(k0 * k2, det);
  if (!(k0 > 0.0f && k2 > 0.0f && det > 0.0f && delta < 0.25f)) {
    s.regular = false;
    return s;
  }
  const float m = 0.02f + 1e-6f * (fabsf(cx) + fabsf(cy) + extent);
  const float ik0 = __fdividef(1.0f, k0), slope = __fdividef(k1, k2), x2 = __fdividef(k2, det);
  const float y0 = (float)ty * ts - cy, y1 = y0 + ts;
  int a0 = 0, b0 = -1, a1 = 0, b1 = -1;
#pragma unroll
  for (int wide = 1; wide >= 0; --wide) {
    const float grow = wide ? m : -m;
    const float level = (2.0f * thr) * (wide ? 1.0f + delta : 1.0f - delta);
    const float lo = y0 - grow, hi = y1 + grow, top = k0 * level;
    const float nearest = fminf(fmaxf(0.0f, lo), hi);
    if (!(top >= det * nearest * nearest)) break;  // the row misses the support
    const float yr = slope * sqrt_approx(level * x2);
    const float dr = fminf(fmaxf(-yr, lo), hi), dl = fminf(fmaxf(yr, lo), hi);
    const float xr = cx + (sqrt_approx(fmaxf(top - det * dr * dr, 0.0f)) - k1 * dr) * ik0 + grow;
    const float xl = cx - (sqrt_approx(fmaxf(top - det * dl * dl, 0.0f)) + k1 * dl) * ik0 - grow;
    if (wide) {
      a0 = max((int)floorf(xl * inv), x0);
      b0 = min((int)floorf(xr * inv), x1);
    } else if (xl <= xr) {
      a1 = max((int)floorf(xl * inv), a0);
      b1 = min((int)floorf(xr * inv), b0);
    }
  }
  if (a0 > b0) return s;
  const bool core = a1 <= b1;
  int hits = core ? b1 - a1 + 1 : 0;
  if (b0 - a0 + 1 - hits > 8) {
    s.regular = false;
    return s;
  }
  s.first = core ? a1 : b0 + 1;
  s.last = core ? b1 : a0 - 1;
  for (int t = a0; t <= b0; ++t) {
    if (core && t == a1) {
      t = b1;
      continue;
    }
    if (tile_rect_test(cx, cy, k0, k1, k2, thr, t, ty, ts)) {
      s.first = min(s.first, t);
      s.last = max(s.last, t);
      ++hits;
    }
  }
  if (hits == 0) {
    s.first = 1;
    s.last = 0;
  } else {
    s.regular = s.last - s.first + 1 == hits;
  }
  return s;
}

// Per-warp tables of the projection's cooperative tile count: the splat
// parameters of the tile test, the box, and the inclusive box-tile counts.
struct CountShared {
  float f[8][kBlock / 32][32];     // cx, cy, conic a, b, c, threshold, rx, ry
  uint32_t u[5][kBlock / 32][32];  // box x0, y0, width, box index of the centre tile (or ~0), wrap
  uint32_t incl[kBlock / 32][32];
  uint32_t cnt[kBlock / 32][32];
};

// The lane whose run of an inclusive scan holds j (the scan's total is above j).
__device__ __forceinline__ uint32_t find_owner(const uint32_t* incl, uint32_t j) {
  uint32_t owner = 0;
#pragma unroll
  for (uint32_t step = 16; step >= 1; step >>= 1)
    if (incl[owner + step - 1] <= j) owner += step;
  return owner;
}

__device__ __forceinline__ uint32_t warp_inclusive(uint32_t v) {
  const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= (uint32_t)d) v += y;
  }
  return v;
}

// Counts the tiles of every lane's box (nbox tiles in rows rows) that pass the
// reference's tile test, with the warp's lanes spread over the union of the
// 32 boxes instead of each lane walking its own. Small boxes share
// rounds of 32 tiles, in row-major order; the centre's tile (`centre`, box
// index u[3]) counts without a test. Boxes of kRowBox tiles or more share rounds
// of 32 rows. Boxes those cannot take (*irregular), and wide ones along a
// periodic axis, are walked tile by tile by the whole warp, one at a time.
// Must be called by all 32 lanes; a lane with nbox == 0 contributes nothing.
// Returns the lane's count.
template <bool PERIODIC>
__device__ __forceinline__ uint32_t count_tiles_warp(CountShared& sm, uint32_t nbox, uint32_t rows, bool centre,
                                                     float vw, float vh, uint32_t axis, float ts, float inv,
                                                     bool* irregular) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const bool by_rows = !PERIODIC && nbox >= kRowBox;
  bool wide = PERIODIC && nbox >= kWideBox;
  const uint32_t walk = centre ? nbox - 1u : nbox;  // the tile walks skip the centre's tile
  const uint32_t incl = warp_inclusive(wide || by_rows ? 0u : walk);
  sm.incl[warp][lane] = incl;
  sm.cnt[warp][lane] = 0u;
  __syncwarp();
  const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
  for (uint32_t j0 = 0; j0 < total; j0 += 32) {
    const uint32_t j = j0 + lane;
    const bool valid = j < total;
    const uint32_t owner = find_owner(sm.incl[warp], j);
    bool hit = false;
    if (valid) {
      const uint32_t bw = sm.u[2][warp][owner];
      uint32_t k = j - (owner ? sm.incl[warp][owner - 1] : 0u);
      k += k >= sm.u[3][warp][owner] ? 1u : 0u;
      const uint32_t by = k / bw, bx = k - by * bw;
      hit = tile_hit<PERIODIC>(sm.f[0][warp][owner], sm.f[1][warp][owner], sm.f[2][warp][owner],
                              sm.f[3][warp][owner], sm.f[4][warp][owner], sm.f[5][warp][owner],
                              sm.f[6][warp][owner], sm.f[7][warp][owner],
                              box_column<PERIODIC>(bx, sm.u[0][warp][owner], sm.u[4][warp][owner], axis),
                              box_row<PERIODIC>(by, sm.u[1][warp][owner], sm.u[4][warp][owner], axis), vw, vh, axis, ts);
    }
    const uint32_t hits = __ballot_sync(0xffffffffu, hit);
    const uint32_t same = __match_any_sync(0xffffffffu, valid ? owner : 32u + lane);
    if (valid && lane == 31u - (uint32_t)__clz(same)) sm.cnt[warp][owner] += __popc(hits & same);
  }
  __syncwarp();
  uint32_t cnt = sm.cnt[warp][lane] + (centre && !by_rows ? 1u : 0u);
  if (!PERIODIC && __any_sync(0xffffffffu, by_rows)) {
    // Rounds of 32 box rows.
    const uint32_t rincl = warp_inclusive(by_rows ? rows : 0u);
    sm.incl[warp][lane] = rincl;
    sm.cnt[warp][lane] = 0u;
    __syncwarp();
    const uint32_t rtotal = __shfl_sync(0xffffffffu, rincl, 31);
    for (uint32_t j0 = 0; j0 < rtotal; j0 += 32) {
      const uint32_t j = j0 + lane;
      if (j < rtotal) {
        const uint32_t owner = find_owner(sm.incl[warp], j);
        const uint32_t row = j - (owner ? sm.incl[warp][owner - 1] : 0u);
        const int x0 = (int)sm.u[0][warp][owner];
        const RowSpan r = row_span(sm.f[0][warp][owner], sm.f[1][warp][owner], sm.f[2][warp][owner],
                                   sm.f[3][warp][owner], sm.f[4][warp][owner], sm.f[5][warp][owner],
                                   (int)(sm.u[1][warp][owner] + row), x0, x0 + (int)sm.u[2][warp][owner] - 1, vw + vh,
                                   ts, inv);
        // The sign bit marks a box that needs the tile walk.
        if (!r.regular) atomicOr(&sm.cnt[warp][owner], 0x80000000u);
        else if (r.last >= r.first) atomicAdd(&sm.cnt[warp][owner], (uint32_t)(r.last - r.first + 1));
      }
    }
    __syncwarp();
    if (by_rows) {
      cnt = sm.cnt[warp][lane];
      wide = (cnt >> 31) != 0u;
    }
  }
  *irregular = wide;
  // The whole warp walks one box, 32 tiles a step.
  uint32_t wide_lanes = __ballot_sync(0xffffffffu, wide);
  while (wide_lanes) {
    const uint32_t w = (uint32_t)__ffs(wide_lanes) - 1u;
    wide_lanes &= wide_lanes - 1u;
    // The owner's parameters are read from the warp's table at each step
    // (broadcast loads) rather than held in registers across the walk.
    const volatile float(*vf)[kBlock / 32][32] = sm.f;
    const volatile uint32_t(*vu)[kBlock / 32][32] = sm.u;
    const uint32_t n = __shfl_sync(0xffffffffu, walk, w);
    uint32_t sum = 0;
    for (uint32_t j0 = 0; j0 < n; j0 += 32) {
      uint32_t k = j0 + lane;
      bool hit = false;
      if (k < n) {
        k += k >= vu[3][warp][w] ? 1u : 0u;
        const uint32_t bw = vu[2][warp][w];
        const uint32_t by = k / bw, bx = k - by * bw;
        hit = tile_hit<PERIODIC>(vf[0][warp][w], vf[1][warp][w], vf[2][warp][w], vf[3][warp][w], vf[4][warp][w],
                                vf[5][warp][w], vf[6][warp][w], vf[7][warp][w],
                                box_column<PERIODIC>(bx, vu[0][warp][w], vu[4][warp][w], axis),
                                box_row<PERIODIC>(by, vu[1][warp][w], vu[4][warp][w], axis), vw, vh, axis, ts);
      }
      sum += __popc(__ballot_sync(0xffffffffu, hit));
    }
    if (lane == w) cnt = sum + (centre ? 1u : 0u);
  }
  return cnt;
}

// GROUPED: some group holds several views (decode once, before the view
// loop); otherwise every group is one view and the decode stays inside the
// per-view chain, after the object tests, where it costs fewest registers.
// VIS: also write the number of visible splats of each 32 items (vis8) and
// fold the visible keys into *key_min, *key_max (the fused front's
// compaction and its choice of sort passes).
// Must be called by all kBlock threads; s_group, s_count are the block's.
template <bool FP64, bool GROUPED, bool FAST_SH, bool PERIODIC, bool VIS>
__device__ __forceinline__ void project_block(uint32_t block, const BatchView& b, const PassOptions& o,
                                              const float* s_snorm, uint32_t& s_group, CountShared& s_count,
                                              float4* __restrict__ mean_out, float4* __restrict__ conic_out,
                                              float4* __restrict__ color_out, uint32_t* __restrict__ count_out,
                                              uint32_t* __restrict__ key_out, float4* __restrict__ rec_out,
                                              float4* __restrict__ erec_out, uint8_t* vis8, uint32_t* key_min,
                                              uint32_t* key_max) {
  if (threadIdx.x == 0) s_group = find_view(b.group_block, b.ngroups, block);
  __syncthreads();
  const uint32_t g = s_group;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t gid = (block - __ldg(b.group_block + g)) * kBlock + threadIdx.x;  // ordinal in each view
  const uint32_t v_first = __ldg(b.group_view + g);
  const uint32_t v_end = GROUPED ? __ldg(b.group_view + g + 1) : v_first + 1u;

  // Decode the splat once for every view of the group (the views share the
  // packed scene, so the active tail, means, shape and rotation are common).
  bool live = false;
  uint32_t slot = 0;
  float4 mo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), so = mo, q = mo;
  m3 local = {};
  {
    const ViewDesc& v = b.views[v_first];
    do {
      if (gid >= v.active) break;  // padding up to the view's next block boundary
      slot = __ldg(v.sh + (size_t)v.count * v.C + gid);
      if (slot >= v.count) break;  // out-of-range tail entries never draw
      mo = __ldg(v.means + slot);
      if (mo.w < 0.0f) break;  // empty slot (ProjectionStage.ts:408-410)
      if (GROUPED) {
        so = decode_scale_opacity(__ldg(v.shape + slot));
        q = decode_rotation(__ldg(v.rot + slot));
        local = local_covariance(so, q);
      }
      live = true;
    } while (false);
  }

  for (uint32_t vi = v_first; vi < v_end; ++vi) {
    const ViewDesc& v = b.views[vi];
    const uint32_t item = v.item_base + gid;
    const float vw = v.vw, vh = v.vh;
    float4 mo4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    uint32_t cnt = 0, key = kInvisibleKey, nbox = 0, rows = 0;
    bool centre = false, irregular = false;
    Projected pr = {};
    float op = 0.0f, rx = 0.0f, ry = 0.0f, thr = 0.0f;
    float ddx = 0.0f, ddy = 0.0f, ddz = 0.0f;  // positionLocal - cameraLocal
    // Project and cull; a splat that survives gets its tile box.
    do {
      if (!live) break;
      const uint32_t obj = (uint32_t)mo.w;
      if (obj >= v.object_count) break;  // unwritten object rows are zero
      const float* ot = v.objects + 40 * (size_t)obj;
      if (!(__ldg(ot + 36) > 0.0f)) break;  // object visibility (:445-450)
      if (!GROUPED) {
        so = decode_scale_opacity(__ldg(v.shape + slot));
        q = decode_rotation(__ldg(v.rot + slot));
      }
      float mv[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) mv[i] = __ldg(ot + 16 + i);
      const float camx = __ldg(ot + 32), camy = __ldg(ot + 33), camz = __ldg(ot + 34);
      ddx = mo.x - camx; ddy = mo.y - camy; ddz = mo.z - camz;
      // view = modelView * (p, 1) (:479-482); the FP64 form evaluates it in
      // double so far-origin coordinates do not cancel against the translation.
      double vxd = 0.0, vyd = 0.0, vzd = 0.0;
      float vx, vy, vz;
      if (FP64) {
        // A product of two floats is exact in double, so a fused multiply-add
        // rounds like the product and the sum; the FP64 unit (2 lanes per SM)
        // is what this form waits for.
        const double px = mo.x, py = mo.y, pz = mo.z;
        vxd = __fma_rn((double)mv[8], pz, __fma_rn((double)mv[4], py, (double)mv[0] * px)) + (double)mv[12];
        vyd = __fma_rn((double)mv[9], pz, __fma_rn((double)mv[5], py, (double)mv[1] * px)) + (double)mv[13];
        vzd = __fma_rn((double)mv[10], pz, __fma_rn((double)mv[6], py, (double)mv[2] * px)) + (double)mv[14];
        vx = (float)vxd; vy = (float)vyd; vz = (float)vzd;
      } else {
        vx = ((mv[0] * mo.x + mv[4] * mo.y) + mv[8] * mo.z) + mv[12] * 1.0f;
        vy = ((mv[1] * mo.x + mv[5] * mo.y) + mv[9] * mo.z) + mv[13] * 1.0f;
        vz = ((mv[2] * mo.x + mv[6] * mo.y) + mv[10] * mo.z) + mv[14] * 1.0f;
      }
      m3 l2v;
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int r = 0; r < 3; ++r) l2v.m[c][r] = mv[4 * c + r];
      const m3 cv = view_covariance(GROUPED ? local : local_covariance(so, q), l2v);
      float P[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) P[i] = v.P[i];
      pr = project({vx, vy, vz}, cv, P, vw, vh, v.vnear, v.vfar, o.filter);
      if (FP64) {
        // Near-singular in FP32 (tiny anti-aliasing factor, high condition
        // number, or rejected past the depth test): redo the chain in double.
        const float cond_num = (pr.cov_x + pr.cov_z) * (pr.cov_x + pr.cov_z);
        const bool redo = !pr.ok ? (-vz > v.vnear && -vz < v.vfar)
                                 : (pr.orig_det < 1e-2f * pr.det || !(cond_num <= 4e3f * pr.det));
        // The redo reads the model-view and projection rows from global memory
        // (the same values as mv and P), so neither array needs a stack copy.
        if (redo) pr = project_fp64(vxd, vyd, vzd, so, q, ot + 16, v.P, vw, vh, v.vnear, v.vfar, o.filter);
      }
      if (!pr.ok) break;
      op = clampf(so.w, 0.0f, 1.0f);
      if (o.antialias == 0u) op = op * sqrtf(clampf(pr.orig_det / pr.det, 0.0f, 1.0f));
      if (op < (float)(1.0 / 255.0) || op != op) break;
      thr = gsdm::logf_(op * 255.0f);
      const float ex = sqrtf((thr * 2.0f) * clampf(pr.cov_x, 1e-12f, 1e4f));
      const float ey = sqrtf((thr * 2.0f) * clampf(pr.cov_z, 1e-12f, 1e4f));
      rx = ceilf(ex);
      ry = ceilf(ey);
      if (rx <= 0.0f || ry <= 0.0f) break;
      const float bminx = pr.cx - rx, bminy = pr.cy - ry, bmaxx = pr.cx + rx, bmaxy = pr.cy + ry;
      if ((o.axis != 1u && (bmaxx < 0.0f || bminx >= vw)) || (o.axis != 2u && (bmaxy < 0.0f || bminy >= vh)))
        break;
      if (o.subpixel != 0u &&
          !subpixel_has_sample(pr.cx, pr.cy, pr.conic_x, pr.conic_y, pr.conic_z, thr, ex, ey, (uint32_t)vw,
                               (uint32_t)vh, o.axis)) {
        mo4 = make_float4(pr.cx, pr.cy, pr.depth, -1.0f);  // subpixel marker (:572-587)
        break;
      }
      const TileBox box = tile_box<PERIODIC>(pr.cx, pr.cy, rx, ry, vw, vh, (int)v.tiles_x, (int)v.tiles_y, o);
      const float mtx = (float)((int)v.tiles_x - 1), mty = (float)((int)v.tiles_y - 1);
      nbox = box.bw * box.bh;
      rows = box.bh;
      // The tile holding the centre, when it is on screen, lies in the box
      // (the floors are monotone and rx, ry >= 1) and passes the reference's
      // tile test by its centre-inside path (tileContribution.ts:16-59): it
      // counts 1 without a test, and the warp walks the box's other tiles.
      const float fcx = floorf(pr.cx * o.tile_inv), fcy = floorf(pr.cy * o.tile_inv);
      centre = !PERIODIC && fcx >= 0.0f && fcx <= mtx && fcy >= 0.0f && fcy <= mty;
      s_count.u[3][warp][lane] =
          centre ? ((uint32_t)fcy - (uint32_t)box.y0) * box.bw + ((uint32_t)fcx - (uint32_t)box.x0) : 0xffffffffu;
      s_count.f[0][warp][lane] = pr.cx; s_count.f[1][warp][lane] = pr.cy;
      s_count.f[2][warp][lane] = pr.conic_x; s_count.f[3][warp][lane] = pr.conic_y;
      s_count.f[4][warp][lane] = pr.conic_z; s_count.f[5][warp][lane] = thr;
      s_count.f[6][warp][lane] = rx; s_count.f[7][warp][lane] = ry;
      s_count.u[0][warp][lane] = (uint32_t)box.x0; s_count.u[1][warp][lane] = (uint32_t)box.y0;
      s_count.u[2][warp][lane] = box.bw;
      if (PERIODIC) s_count.u[4][warp][lane] = box.wrap;
    } while (false);
    // Tiles passing the tile test (projectionHelpers.ts:223-236), counted by the whole warp.
    cnt = count_tiles_warp<PERIODIC>(s_count, nbox, rows, centre, vw, vh, o.axis, o.tile_px, o.tile_inv, &irregular);
    if (cnt > 0) {
      uint32_t co[16];
      load_sh(v.sh + (size_t)slot * v.C, v.degree, co);
      // viewDirection = normalize(positionLocal - cameraLocal) (:469), which
      // feeds only the colour: the reference's quotients for the EXACT form,
      // a reciprocal square root (2 ulp) for the fast forms' colour.
      const float dd2 = (ddx * ddx + ddy * ddy) + ddz * ddz;
      f3 vdir;
      if (FAST_SH) {
        const float r = rsqrtf(dd2);
        vdir = {ddx * r, ddy * r, ddz * r};
      } else {
        const float dlen = sqrtf(dd2);
        vdir = {ddx / dlen, ddy / dlen, ddz / dlen};
      }
      const f3 col = eval_sh_any<FAST_SH>(v.degree, co, vdir, s_snorm);
      mo4 = make_float4(pr.cx, pr.cy, pr.depth, op);
      conic_out[item] = make_float4(pr.conic_x, pr.conic_y, pr.conic_z, rx + ry * 512.0f);
      // Emission record: what the emission reads per depth rank, in one
      // 32-byte gather (layout in pass_common.cuh).
      erec_out[2 * (size_t)item] = make_float4(pr.cx, pr.cy, pr.conic_x, pr.conic_y);
      erec_out[2 * (size_t)item + 1] = make_float4(pr.conic_z, thr, rx + ry * 512.0f, irregular ? 1.0f : 0.0f);
      color_out[item] = make_float4(col.x, col.y, col.z, __uint_as_float(slot ^ kActiveTag));
      if (rec_out) {
        // Packed raster record of the fast forms (layout in pass_common.cuh).
        const float log2op = __log2f(op);
        const __half2 rg = __floats2half2_rn(col.x, col.y);
        const __half2 bl = __floats2half2_rn(col.z, fminf(log2op, kLog2MaxAlpha));
        rec_out[2 * (size_t)item] = make_float4(pr.cx, pr.cy, -0.5f * kLog2e * pr.conic_x, -kLog2e * pr.conic_y);
        rec_out[2 * (size_t)item + 1] =
            make_float4(-0.5f * kLog2e * pr.conic_z, log2op, __uint_as_float(*reinterpret_cast<const uint32_t*>(&rg)),
                        __uint_as_float(*reinterpret_cast<const uint32_t*>(&bl)));
      }
      if (o.depth_mode == 0u) {
        key = __float_as_uint(pr.depth);  // visibility.ts:139
      } else {
        float t = clampf((pr.depth - v.vnear) / (v.vfar - v.vnear), 0.0f, 1.0f);
        key = (uint32_t)gsdm::round_even_small(t * 65535.0f);  // visibility.ts:140-144
      }
    }
    mean_out[item] = mo4;
    count_out[item] = cnt;
    key_out[item] = key;
    if (VIS) {
      const uint32_t vis = __ballot_sync(0xffffffffu, key != kInvisibleKey);
      if (lane == 0) vis8[item >> 5] = (uint8_t)__popc(vis);
      if (vis) {
        const uint32_t lo = __reduce_min_sync(0xffffffffu, key);
        const uint32_t hi = __reduce_max_sync(0xffffffffu, key == kInvisibleKey ? 0u : key);
        if (lane == 0) {
          // Most warps lie inside the range seen so far.
          if (lo < *(volatile uint32_t*)key_min) atomicMin(key_min, lo);
          if (hi > *(volatile uint32_t*)key_max) atomicMax(key_max, hi);
        }
      }
    }
  }
}

}  // namespace gs
