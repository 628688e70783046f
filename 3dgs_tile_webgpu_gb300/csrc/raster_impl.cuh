// Front-to-back tile rasterizer body (src/renderer/pipeline/TileRasterizer.ts:414-805,
// storeFinalPixel :930-964, finalizeGaussianDepth.ts:18-68, chunk split
// rasterChunks.ts:3-99 and composite TileRasterizer.ts:807-902).
//
// One 256-thread block per 16x16 tile, one pixel per thread, lanes mapped to
// pixels in the reference's compact Morton order (rasterHelpers.ts:3-12), so
// warp w owns an 8x4 patch of the tile. Blocks take tiles from a work list
// ordered heaviest first, so long tiles start early and do not form a tail.
// Each batch of 256 sorted records is gathered into shared memory once.
// While staging, the thread that loads a record also tests the splat's
// support box against the eight warp patches and stores an 8-bit mask; each
// warp then walks only the records whose bit is set (ballot + find-first-set,
// ascending, so front-to-back order holds). The culling is conservative: a
// skipped (pixel, splat) pair is one where the per-pixel test rejects the
// splat anyway, so the result is unchanged. The block leaves the tile when no
// pixel is still accumulating (__syncthreads_or), a warp leaves a batch when
// all its pixels are done (__all_sync).
//
// Tiles holding more than `chunk` samples are evaluated as the reference's
// exact chunks: every chunk starts at transmittance 1 and its partial
// (colour, transmittance, depth) is composited in order; the block runs the
// chunks of its tile one after another and stops once the composite
// transmittance falls below the threshold, which yields exactly the composite
// of the reference's parallel chunk tasks.
//
// Arithmetic: the reference's expressions and tests in their order, with the
// deterministic exp/log (ExactMath); bit-identical to the CPU restatement when
// the translation unit is built with --fmad=false. The fast forms
// (raster_half2.cuh: FP32 and packed half2) share the helpers at the end of this
// file: the packed-record decoding and the exact ellipse-patch test.
#pragma once

#include <cuda_fp16.h>

#include "detmath.h"
#include "pass_common.cuh"

namespace gs {

constexpr float kLog2e = 1.4426950408889634f;

struct ExactMath {
  static constexpr bool kExact = true;
  static __device__ __forceinline__ float exp(float x) { return gsdm::expf_(x); }
  static __device__ __forceinline__ float log(float x) { return gsdm::logf_(x); }
};

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ uint32_t morton_compact(uint32_t v) {
  uint32_t r = v & 0x55555555u;
  r = (r | (r >> 1)) & 0x33333333u;
  r = (r | (r >> 2)) & 0x0f0f0f0fu;
  r = (r | (r >> 4)) & 0x00ff00ffu;
  r = (r | (r >> 8)) & 0x0000ffffu;
  return r;
}

__device__ __forceinline__ float rclamp(float x, float lo, float hi) {
  float y = x < lo ? lo : x;
  return y > hi ? hi : y;
}

// Frame values the rasterizer reads per sample, held in registers.
struct RasterFrame {
  float vw, vh, t_threshold;
  uint32_t axis;
};

// tileContribution.ts:66-82 gaussian_boundary_delta.
template <bool PERIODIC>
__device__ __forceinline__ void boundary_delta(float pxc, float pyc, float cx, float cy, float ca, float cb,
                                               float cc, const RasterFrame& f, float* dx, float* dy) {
  if (!PERIODIC) {
    *dx = pxc - cx;
    *dy = pyc - cy;
    return;
  }
  float ccx = cx, ccy = cy;
  if (f.axis == 1u) ccx = ccx - floorf(cx / f.vw) * f.vw;
  if (f.axis == 2u) ccy = ccy - floorf(cy / f.vh) * f.vh;
  float ddx = pxc - ccx, ddy = pyc - ccy;
  if (f.axis == 1u) {
    float opt = (-cb * ddy) / ca;
    ddx = ddx - floorf((ddx - opt) / f.vw + 0.5f) * f.vw;
  } else {
    float opt = (-cb * ddx) / cc;
    ddy = ddy - floorf((ddy - opt) / f.vh + 0.5f) * f.vh;
  }
  *dx = ddx;
  *dy = ddy;
}

// The centre's image inside the period of a periodic axis (the expressions of
// boundary_delta, so the same bits).
__device__ __forceinline__ float canonical_x(float cx, const RasterFrame& f) {
  return f.axis == 1u ? cx - floorf(cx / f.vw) * f.vw : cx;
}
__device__ __forceinline__ float canonical_y(float cy, const RasterFrame& f) {
  return f.axis == 2u ? cy - floorf(cy / f.vh) * f.vh : cy;
}

// Whether a splat whose support reaches h along the periodic axis shows at
// most one image to the pixels of any patch (at most 16 pixels long). The
// pixels p of a patch that pass the alpha test have |p - centre - k period|
// <= h for the image k that boundary_delta picks; with 2 h + 18 below the
// period, every such k is the image nearest to the patch's middle. Any other
// pixel of the patch fails the test at every image, boundary_delta's
// minimising one included.
__device__ __forceinline__ bool single_image(float h, const RasterFrame& f) {
  return 2.0f * h + 18.0f < (f.axis == 1u ? f.vw : f.vh);
}
__device__ __forceinline__ float nearest_image(float canon, float middle, float period) {
  return rintf((middle - canon) / period);
}

struct PixelAcc {
  float r, g, b, t, d;
};

// Shared batch of the exact form (NB records: one per thread of the tile's
// block, at most 256): geo = (cx, cy, opacity, threshold), con = (a, b, c,
// depth), colour, and the warp-patch masks (bit w: warp w's 8x4 patch can be
// reached).
template <int NT>
struct Batch {
  static constexpr int NB = NT < 256 ? NT : 256;
  float4 geo[NB];
  float4 con[NB];
  float4 col[NB];
  uint32_t mask[NB];
};

constexpr float kLog2MinAlpha = -7.99435329f;  // log2(1/255)
constexpr float kLog2MaxAlpha = -0.01449957f;  // log2(0.99)

// Which of the tile's NW 8x4 warp patches can hold a pixel centre inside
// the splat's support {q(d) <= 2 threshold}. Warp w's lanes are the Morton
// indices 32 w .. 32 w + 31, so its patch starts at the Morton decode of
// 32 w. Conservative: the support's
// bounding box is widened by 5 % + 0.25 px, far beyond the rounding of the
// per-pixel evaluation for conics whose condition number is below 4e4 (the
// 0.3 px^2 filter bounds it near 3.3e4); worse-conditioned splats and
// non-finite values keep every bit set. With a periodic boundary the box is
// tested at the splat's image nearest to each patch, the only one a pixel of
// the patch can see while the extent is below half the period
// (nearest_image); larger splats keep every bit set.
template <int NW>
__device__ __forceinline__ uint32_t patch_mask(float cx, float cy, float ca, float cb, float cc, float thr,
                                               float tile_x0, float tile_y0, const RasterFrame& f) {
  constexpr uint32_t kAll = NW >= 32 ? 0xffffffffu : (1u << NW) - 1u;
  const float det = ca * cc - cb * cb;
  const float tr = ca + cc;
  if (!(det > 0.0f) || !(tr * tr <= 4e4f * det) || !(thr >= 0.0f)) return kAll;
  const float q = 2.0f * thr;
  const float hx = sqrtf(q * cc / det) * 1.05f + 0.25f;
  const float hy = sqrtf(q * ca / det) * 1.05f + 0.25f;
  if (!(hx < 1e30f) || !(hy < 1e30f)) return kAll;
  if (f.axis != 0u && !single_image(f.axis == 1u ? hx : hy, f)) return kAll;
  const float ccx = canonical_x(cx, f), ccy = canonical_y(cy, f);
  uint32_t m = 0;
#pragma unroll
  for (uint32_t w = 0; w < (uint32_t)NW; ++w) {
    const float x0 = tile_x0 + (float)morton_compact(32u * w) + 0.5f;
    const float y0 = tile_y0 + (float)morton_compact(16u * w) + 0.5f;
    float px = cx, py = cy;
    if (f.axis == 1u) px = ccx + nearest_image(ccx, x0 + 3.5f, f.vw) * f.vw;
    if (f.axis == 2u) py = ccy + nearest_image(ccy, y0 + 1.5f, f.vh) * f.vh;
    const bool hit = px + hx >= x0 && px - hx <= x0 + 7.0f && py + hy >= y0 && py - hy <= y0 + 3.0f;
    m |= hit ? (1u << w) : 0u;
  }
  return m;
}

// One (pixel, splat) step of the front-to-back blend (TileRasterizer.ts:616-707).
// Returns true when the pixel is done (transmittance below the threshold).
template <class M, bool PERIODIC, int NT>
__device__ __forceinline__ bool blend_one(const Batch<NT>& sb, uint32_t j, float pxc, float pyc, const RasterFrame& f,
                                          PixelAcc& a, uint32_t* blended) {
  const float4 g = sb.geo[j];
  const float4 c = sb.con[j];
  static_assert(M::kExact, "the fast form blends in blend_range_fast");
  float dx, dy;
  boundary_delta<PERIODIC>(pxc, pyc, g.x, g.y, c.x, c.y, c.z, f, &dx, &dy);
  const float power = ((c.x * (dx * dx) + ((c.y * 2.0f) * dx) * dy) + c.z * (dy * dy)) * -0.5f;
  if (power > 0.0f || power < -g.w) return false;
  const float alpha = rclamp(g.z * M::exp(power), 0.0f, 0.99f);
  if (alpha < (float)(1.0 / 255.0)) return false;
  const float4 col = sb.col[j];
  const float contrib = a.t * alpha;
  a.r = a.r + col.x * contrib;
  a.g = a.g + col.y * contrib;
  a.b = a.b + col.z * contrib;
  a.d = a.d + c.w * contrib;
  a.t = a.t * (1.0f - alpha);
  if (blended) ++*blended;
  return a.t < f.t_threshold;
}

struct RasterCounters {
  uint32_t checked, blended;
};

// Blend samples [s0, s1) of the tile into `a` (block-cooperative; every thread
// of the block must call it). `done` marks pixels that take no more samples.
// With STATS, `cnt` receives the reference's per-pixel counters: samples
// examined until done (TileRasterizer.ts:617) and samples blended (:702).
template <class M, bool PERIODIC, bool STATS, int NT>
__device__ __forceinline__ void blend_range(uint32_t begin, uint32_t source_count, uint32_t raster_count,
                                            uint32_t s0, uint32_t s1, bool capped, const uint32_t* __restrict__ ids,
                                            const float4* __restrict__ mean, const float4* __restrict__ conic,
                                            const float4* __restrict__ color, const RasterFrame& f, float tile_x0,
                                            float tile_y0, float pxc, float pyc, bool done, PixelAcc& a,
                                            Batch<NT>& sb, RasterCounters& cnt) {
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  const bool counting = STATS && !done;
  uint32_t stop = s1;  // sample index after which this pixel stopped
  constexpr uint32_t NB = (uint32_t)Batch<NT>::NB;
  for (uint32_t b = s0; b < s1; b += NB) {
    if (!__syncthreads_or(!done)) break;
    const uint32_t i = b + t;
    if (t < NB && i < s1) {
      uint32_t src = i;
      if (capped) src = (uint32_t)floorf((((float)i + 0.5f) * (float)source_count) / (float)raster_count);
      const uint32_t g = __ldg(ids + begin + src);
      const float4 m = __ldg(mean + g);
      const float4 c = __ldg(conic + g);
      const float thr = M::log(m.w * 255.0f);
      sb.geo[t] = make_float4(m.x, m.y, m.w, thr);
      sb.con[t] = make_float4(c.x, c.y, c.z, m.z);
      sb.col[t] = __ldg(color + g);
      sb.mask[t] = patch_mask<NT / 32>(m.x, m.y, c.x, c.y, c.z, thr, tile_x0, tile_y0, f);
    }
    __syncthreads();
    const uint32_t n = min(NB, s1 - b);
    for (uint32_t c0 = 0; c0 < n; c0 += 32) {
      if (__all_sync(0xffffffffu, done)) break;
      const uint32_t k = c0 + lane;
      uint32_t bits = __ballot_sync(0xffffffffu, k < n && ((sb.mask[k] >> warp) & 1u));
      while (bits) {
        const uint32_t j = c0 + (uint32_t)(__ffs(bits) - 1);
        bits &= bits - 1u;
        if (!done) {
          done = blend_one<M, PERIODIC, NT>(sb, j, pxc, pyc, f, a, STATS ? &cnt.blended : nullptr);
          if (STATS && done) stop = b + j + 1;
        }
      }
    }
  }
  __syncthreads();  // shared batch buffers are free again
  if (counting) cnt.checked += stop - s0;
}

// The conic (a, b, c) back from a packed raster record's scaled terms.
__device__ __forceinline__ float4 raw_conic(const float4& r0, const float4& r1) {
  constexpr float kNeg2Ln2 = -1.38629436f;  // 1 / (-1/2 log2 e)
  constexpr float kNegLn2 = -0.693147181f;  // 1 / (-log2 e)
  return make_float4(r0.z * kNeg2Ln2, r0.w * kNegLn2, r1.x * kNeg2Ln2, 0.0f);
}

// The quadratic of a packed record, for culling: F = A dx^2 + B dx dy + C dy^2
// (the scaled conic, F >= 0), and whether a pixel can pass the splat's
// alpha >= 1/255 test, F(d) <= R = log2(255 opacity). `limit` carries a margin
// (1% of R + 0.01) that exceeds the rounding of both evaluations for conics
// whose condition number is below about 1e4; worse-conditioned splats are
// `always` in reach.
struct ReachTest {
  float A, B, C, ia, ic, limit;
  bool always;
};
__device__ __forceinline__ ReachTest reach_test(float ap, float bp, float cp, float log2op) {
  ReachTest t;
  t.A = -ap; t.B = -bp; t.C = -cp;
  const float det4 = 4.0f * t.A * t.C - t.B * t.B;  // 4 det of [[A, B/2], [B/2, C]]
  const float tr = t.A + t.C;
  t.always = !(t.A > 0.0f) || !(t.C > 0.0f) || !(det4 > 0.0f) || !(tr * tr <= 1e4f * det4);
  t.ic = __fdividef(-0.5f * t.B, t.C);
  t.ia = __fdividef(-0.5f * t.B, t.A);
  t.limit = fmaf(log2op + 7.99435329f, 1.01f, 0.01f);
  return t;
}

// One side of the rectangle [lo, hi] x [..] seen from the centre: the offset
// nearest to the centre along that axis, and what F's minimum along it needs.
struct ReachEdge {
  float lo, hi;         // the rectangle's offsets along this axis
  float best, lin, sq;  // unconstrained minimiser of the other axis, B x, A x^2
};
__device__ __forceinline__ ReachEdge reach_edge(float centre, float x0, float w, float slope, float lin, float sq) {
  ReachEdge e;
  e.lo = x0 - centre;
  e.hi = e.lo + w;
  const float x = fminf(fmaxf(0.0f, e.lo), e.hi);
  e.best = slope * x;
  e.lin = lin * x;
  e.sq = sq * x * x;
  return e;
}
// Whether the rectangle x-side ex by y-side ey holds a point in reach. F is
// convex with its minimum, 0, at the centre, so over a rectangle that does not
// hold the centre its minimum lies on an edge that faces the centre: the line
// x = nearest x (with y clamped to the rectangle) or y = nearest y. A
// rectangle that holds the centre has 0 on both. (All four edges: the
// rasterizer took 3218 us instead of 3100 for 16 views of 3M splats at 1080p,
// half2 form, and 367 instead of 350 for one in FP32; a quarter of its
// instructions are this test, and four of five records fail it.)
__device__ __forceinline__ bool reach_rect(const ReachTest& t, const ReachEdge& ex, const ReachEdge& ey) {
  const float dy = fminf(fmaxf(ex.best, ey.lo), ey.hi), dx = fminf(fmaxf(ey.best, ex.lo), ex.hi);
  const float m = fminf(fmaf(fmaf(t.C, dy, ex.lin), dy, ex.sq), fmaf(fmaf(t.A, dx, ey.lin), dx, ey.sq));
  return t.always || !(m > t.limit);  // NaN: reach
}

// Can a pixel centre of the rectangle [x0, x0 + wx] x [y0, y0 + wy] pass the
// splat's alpha test?
__device__ __forceinline__ bool patch_reach(float cx, float cy, float ap, float bp, float cp, float log2op,
                                            float x0, float y0, float wx, float wy) {
  const ReachTest t = reach_test(ap, bp, cp, log2op);
  return reach_rect(t, reach_edge(cx, x0, wx, t.ic, t.B, t.A), reach_edge(cy, y0, wy, t.ia, t.B, t.C));
}

__device__ __forceinline__ bool finite_r(float v) { return v == v && fabsf(v) <= 3.402823e+38f; }

// finalizeGaussianDepth.ts:18-68 with the default nodes (GaussianContextNodes.ts:127-132).
__device__ __forceinline__ float finalize_depth(float wd, float trans, const PassOptions& o, float vnear,
                                                float vfar) {
  float a = 1.0f - trans;
  float out = 0.0f;
  if (a > 0.0f) out = wd / a;
  bool scalar_valid = a > 0.0f && finite_r(wd) && finite_r(out) && out > 0.0f;
  bool valid = scalar_valid && a > o.depth_alpha_threshold;
  float dev = o.invalid_depth;
  if (valid) {
    float enc;
    if (o.depth_encoding == 0u) {
      float vz = -out;
      enc = rclamp(((vnear + vz) * vfar) / ((vfar - vnear) * vz), 0.0f, 1.0f);
    } else {
      enc = out;
    }
    if (finite_r(enc)) dev = enc;
  }
  return dev;
}

// One block of TILE x TILE threads per tile of the batch (in work-list order),
// lanes on pixels in the Morton order (warp w: an 8x4 patch); the tile's view
// supplies its viewport and targets.
template <class M, bool PERIODIC, bool STATS, int TILE>
__global__ void __launch_bounds__(TILE * TILE, TILE == 32 ? 1 : 768 / (TILE * TILE))
    k_raster(const uint32_t* __restrict__ tile_offsets,
                                                   const uint32_t* __restrict__ order,
                                                   const uint32_t* __restrict__ ids,
                                                   const float4* __restrict__ mean,
                                                   const float4* __restrict__ conic,
                                                   const float4* __restrict__ color, BatchView bv, PassOptions o,
                                                   Control* __restrict__ ctl) {
  after_previous();
  // Overflow: the reference zeroes the raster dispatch, so nothing is written.
  if (ctl->state[3] != 0u) return;
  constexpr int NT = TILE * TILE;
  __shared__ Batch<NT> sb;
  __shared__ uint32_t s_view;
  __shared__ unsigned long long s_stats[4];
  const uint32_t tile = order ? order[blockIdx.x] : blockIdx.x;
  if (threadIdx.x == 0) s_view = find_view(bv.tile_base, bv.nviews, tile);
  if (STATS && threadIdx.x < 4) s_stats[threadIdx.x] = 0ull;
  __syncthreads();
  const ViewDesc& v = bv.views[s_view];
  const RasterFrame f = {v.vw, v.vh, o.t_threshold, o.axis};
  const uint32_t local = tile - v.tile_base;
  const uint32_t tx = local % v.tiles_x, ty = local / v.tiles_x;
  const uint32_t lx = morton_compact(threadIdx.x), ly = morton_compact(threadIdx.x >> 1);
  const uint32_t px = tx * TILE + lx, py = ty * TILE + ly;
  const uint32_t W = (uint32_t)v.vw, H = (uint32_t)v.vh;
  const bool active = px < W && py < H;
  const uint32_t begin = tile_offsets[tile], end = tile_offsets[tile + 1];
  const uint32_t source_count = end - begin;
  const bool capped = o.max_per_tile != 0u;
  const uint32_t raster_count = capped ? min(source_count, o.max_per_tile) : source_count;
  const uint32_t chunk = o.chunk;
  const bool chunked = chunk != 0u && raster_count > chunk;
  const float pxc = (float)px + 0.5f, pyc = (float)py + 0.5f;
  const float tile_x0 = (float)(tx * TILE), tile_y0 = (float)(ty * TILE);
  PixelAcc a = {0.0f, 0.0f, 0.0f, 1.0f, 0.0f};
  RasterCounters cnt = {0u, 0u};
  if (!chunked) {
    blend_range<M, PERIODIC, STATS, NT>(begin, source_count, raster_count, 0, raster_count, capped, ids, mean,
                                        conic, color, f, tile_x0, tile_y0, pxc, pyc, !active, a, sb, cnt);
  } else {
    const uint32_t nchunk = (raster_count + chunk - 1) / chunk;
    bool finished = !active;
    for (uint32_t ch = 0; ch < nchunk; ++ch) {
      if (!__syncthreads_or(!finished)) break;
      const uint32_t s0 = ch * chunk;
      const uint32_t s1 = min(s0 + chunk, raster_count);
      PixelAcc p = {0.0f, 0.0f, 0.0f, 1.0f, 0.0f};
      blend_range<M, PERIODIC, STATS, NT>(begin, source_count, raster_count, s0, s1, capped, ids, mean, conic,
                                          color, f, tile_x0, tile_y0, pxc, pyc, finished, p, sb, cnt);
      if (!finished) {
        a.r = a.r + p.r * a.t;
        a.g = a.g + p.g * a.t;
        a.b = a.b + p.b * a.t;
        a.d = a.d + p.d * a.t;
        a.t = a.t * p.t;
        if (a.t < f.t_threshold) finished = true;
      }
    }
  }
  if (STATS) {
    // TileRasterizer.ts:749-768: checked, blended, pixels, alpha-stopped.
    if (active) {
      atomicAdd(&s_stats[0], (unsigned long long)cnt.checked);
      atomicAdd(&s_stats[1], (unsigned long long)cnt.blended);
      if (raster_count > 0) {
        atomicAdd(&s_stats[2], 1ull);
        if (a.t < f.t_threshold) atomicAdd(&s_stats[3], 1ull);
      }
    }
    __syncthreads();
    if (threadIdx.x < 4 && s_stats[threadIdx.x]) atomicAdd(&ctl->raster_stats[threadIdx.x], s_stats[threadIdx.x]);
  }
  if (!active) return;
  const float bga = rclamp(o.background[3], 0.0f, 1.0f);
  const float r = a.r + (o.background[0] * a.t) * bga;
  const float g = a.g + (o.background[1] * a.t) * bga;
  const float b = a.b + (o.background[2] * a.t) * bga;
  const float alpha = 1.0f - a.t * (1.0f - bga);
  const size_t off = (size_t)py * W + px;
  if (v.color_half) {
    __half2 lo = __floats2half2_rn(r, g);
    __half2 hi = __floats2half2_rn(b, alpha);
    uint2 w;
    w.x = *reinterpret_cast<uint32_t*>(&lo);
    w.y = *reinterpret_cast<uint32_t*>(&hi);
    reinterpret_cast<uint2*>(v.color)[off] = w;
  } else {
    reinterpret_cast<float4*>(v.color)[off] = make_float4(r, g, b, alpha);
  }
  if (v.depth) v.depth[off] = finalize_depth(a.d, a.t, o, v.vnear, v.vfar);
}

template <class M, int TILE>
void launch_raster_tile(const uint32_t* tile_offsets, const uint32_t* order, const uint32_t* ids,
                        const float4* mean, const float4* conic, const float4* color, const BatchView& b,
                        const PassOptions& o, Control* ctl, bool stats, cudaStream_t st) {
  const bool periodic = o.axis != 0u;
#define GS_RASTER(P, S)                                                                                          \
  launch_after(k_raster<M, P, S, TILE>, b.total_tiles, TILE * TILE, 0, st, tile_offsets, order, ids, mean,         \
               conic, color, b, o, ctl)
  if (periodic) {
    if (stats) GS_RASTER(true, true); else GS_RASTER(true, false);
  } else {
    if (stats) GS_RASTER(false, true); else GS_RASTER(false, false);
  }
#undef GS_RASTER
}

template <class M>
void launch_raster_policy(const uint32_t* tile_offsets, const uint32_t* order, const uint32_t* ids,
                          const float4* mean, const float4* conic, const float4* color, const BatchView& b,
                          const PassOptions& o, Control* ctl, bool stats, cudaStream_t st) {
  if (b.total_tiles == 0) return;
  if (o.tile == 8u)
    launch_raster_tile<M, 8>(tile_offsets, order, ids, mean, conic, color, b, o, ctl, stats, st);
  else if (o.tile == 32u)
    launch_raster_tile<M, 32>(tile_offsets, order, ids, mean, conic, color, b, o, ctl, stats, st);
  else
    launch_raster_tile<M, 16>(tile_offsets, order, ids, mean, conic, color, b, o, ctl, stats, st);
}

}  // namespace gs
