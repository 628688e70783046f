// Kernels whose integer outputs must be bit-identical to the CPU restatement:
// projection + tile count, visibility compaction, the saturating intersection
// scan, intersection emission and tile ranges; plus the bit-exact raster form.
// Built with --fmad=false (see build.py): no multiply-add contraction, so each
// float expression rounds exactly like the CPU restatement.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "emission.cuh"
#include "pass_common.cuh"
#include "projection.cuh"
#include "raster_impl.cuh"
#include "splat_math.cuh"

namespace gs {

// ---------------------------------------------------------------------------
// The projection kernel: a block per 256 ordinals of a view group
// (project_block, projection.cuh).
template <bool FP64, bool GROUPED, bool FAST_SH, bool PERIODIC>
__global__ void __launch_bounds__(kBlock, kProjectBlocksPerSm)
    k_project(BatchView b, PassOptions o, float4* __restrict__ mean_out, float4* __restrict__ conic_out,
              float4* __restrict__ color_out, uint32_t* __restrict__ count_out, uint32_t* __restrict__ key_out,
              float4* __restrict__ rec_out, float4* __restrict__ erec_out) {
  __shared__ float s_snorm[256];
  __shared__ uint32_t s_group;
  __shared__ CountShared s_count;
  s_snorm[threadIdx.x] = snorm8_value(threadIdx.x);
  project_block<FP64, GROUPED, FAST_SH, PERIODIC, false>(blockIdx.x, b, o, s_snorm, s_group, s_count, mean_out,
                                                         conic_out, color_out, count_out, key_out, rec_out, erec_out,
                                                         nullptr, nullptr, nullptr);
}

template <bool FAST_SH>
void launch_project_t(const BatchView& b, const PassOptions& o, float4* mean, float4* conic, float4* color,
                      uint32_t* counts, uint32_t* keys, float4* rec, float4* erec, cudaStream_t st) {
  const bool grouped = b.ngroups < b.nviews;
#define GS_PROJECT(F, G)                                                                                          \
  if (o.axis)                                                                                                     \
    k_project<F, G, FAST_SH, true>                                                                                \
        <<<b.total_blocks, kBlock, 0, st>>>(b, o, mean, conic, color, counts, keys, rec, erec);                   \
  else                                                                                                            \
    k_project<F, G, FAST_SH, false><<<b.total_blocks, kBlock, 0, st>>>(b, o, mean, conic, color, counts, keys, rec, erec)
  if (o.proj_fp64) {
    if (grouped) { GS_PROJECT(true, true); } else { GS_PROJECT(true, false); }
  } else {
    if (grouped) { GS_PROJECT(false, true); } else { GS_PROJECT(false, false); }
  }
#undef GS_PROJECT
}

// The fast raster forms (rec != null) take the fused-multiply-add SH colour;
// EXACT keeps the reference's order.
void launch_project(const BatchView& b, const PassOptions& o, float4* mean, float4* conic, float4* color,
                    uint32_t* counts, uint32_t* keys, float4* rec, float4* erec, cudaStream_t st) {
  if (b.total_blocks == 0) return;  // projection blocks over the view groups
  if (rec) launch_project_t<true>(b, o, mean, conic, color, counts, keys, rec, erec, st);
  else launch_project_t<false>(b, o, mean, conic, color, counts, keys, rec, erec, st);
}

// ---------------------------------------------------------------------------
// Chunked scans (visibility compaction, ordered-count scan): a persistent grid
// of at most `chunks` blocks; chunk c (tickets give launch order) is a
// contiguous run of 256-item units, split into one contiguous slice per warp.
// Phase 1 reduces each warp's slice and publishes the chunk's sum, the block
// adds up the sums of the chunks before its own, and phase 2 walks the slice
// again writing every output with the warp's running offset. A unit is 8 rows
// of 32 consecutive items, so every load and store of a row is one coalesced
// 128-byte access.
//
// A block reads all the sums before its own at once (256 words a round trip
// and thread slot) instead of looking back for a published prefix: the blocks
// end phase 1 together, so prefixes trickle up the chunks one window after the
// other. Look-back / sums: 3M ordinals compaction 25.4 / 24.2 us, scan 30.4 /
// 27.9; 6M 35.1 / 33.2, 52.4 / 50.9; 48M 201 / 198, 357 / 354. What is left is
// the latency of the two phases and the gather of the counts; 6 or 8 blocks per
// SM scan slower (28 -> 31 / 36 us, 51 -> 52 / 59).
constexpr uint32_t kUnit = 256;
constexpr uint32_t kUnitRows = kUnit / 32;
constexpr uint32_t kScanWarps = kBlock / 32;

// The chunks that n items fill, none of them empty (one when n is 0).
__device__ __forceinline__ uint32_t filled_chunks(uint32_t n, uint32_t chunks) {
  return min(chunks, max(n / kUnit + (n % kUnit != 0u), 1u));
}

// Units [w0, w1) of warp `warp` of chunk c.
__device__ __forceinline__ void warp_units(uint32_t n, uint32_t chunks, uint32_t c, uint32_t warp, uint32_t* w0,
                                           uint32_t* w1) {
  const uint32_t units = (uint32_t)(((uint64_t)n + kUnit - 1) / kUnit);
  const uint32_t u0 = (uint32_t)((uint64_t)c * units / chunks), u1 = (uint32_t)((uint64_t)(c + 1u) * units / chunks);
  *w0 = u0 + (u1 - u0) * warp / kScanWarps;
  *w1 = u0 + (u1 - u0) * (warp + 1u) / kScanWarps;
}

struct ScanShared {
  uint32_t chunk;
  uint32_t warp[kScanWarps];            // sums of the warps' slices
  unsigned long long part[kScanWarps];  // sums of the chunks before, by warp
};

// Called by the whole block with sm.warp filled: publishes chunk c's sum and
// adds up those before it. *run is the warp's exclusive base, *through the sum
// up to and with this chunk, both saturating at 0xffffffff.
__device__ __forceinline__ void chunk_prefix(ScanShared& sm, unsigned long long* status, uint32_t c, uint32_t epoch,
                                             uint32_t limit, uint32_t* err, uint32_t* run, uint32_t* through) {
  constexpr uint32_t kAtOnce = 4;
  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  __syncthreads();
  unsigned long long mine = 0, below = 0, before = 0;
#pragma unroll
  for (uint32_t w = 0; w < kScanWarps; ++w) {
    mine += sm.warp[w];
    below += w < warp ? sm.warp[w] : 0u;
  }
  if (tid == 0) st_status(status + c, epoch, (uint32_t)min(mine, 0xffffffffull));
  for (uint32_t i = tid; i < c; i += kAtOnce * kBlock) {
    unsigned long long v[kAtOnce];
#pragma unroll
    for (uint32_t k = 0; k < kAtOnce; ++k) v[k] = i + k * kBlock < c ? ld_status(status + i + k * kBlock) : 0ull;
#pragma unroll
    for (uint32_t k = 0; k < kAtOnce; ++k)
      if (i + k * kBlock < c) before += wait_status(status + i + k * kBlock, v[k], epoch, limit, err);
  }
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) before += __shfl_xor_sync(0xffffffffu, before, d);
  if ((tid & 31u) == 0u) sm.part[warp] = before;
  __syncthreads();
  before = 0;
#pragma unroll
  for (uint32_t w = 0; w < kScanWarps; ++w) before += sm.part[w];
  *run = (uint32_t)min(before + below, 0xffffffffull);
  *through = (uint32_t)min(before + mine, 0xffffffffull);
}

// Visibility compaction (scan.ts:9-83 + visibility.ts:9-61). Writes
// visibleOffsets, the (depthKey, ordinal) records in ordinal order and the
// visible state.
__global__ void __launch_bounds__(kBlock) k_compact(const uint32_t* __restrict__ keys, uint32_t n,
                                                    uint32_t* __restrict__ vis_off, uint32_t* __restrict__ keys_out,
                                                    uint32_t* __restrict__ vals_out, Control* __restrict__ ctl,
                                                    unsigned long long* __restrict__ status, Epoch ep,
                                                    uint32_t chunks) {
  next_may_launch();
  __shared__ ScanShared sm;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (tid == 0) sm.chunk = atomicAdd(&ctl->tickets[kTicketCompact], 1u);
  __syncthreads();
  const uint32_t c = sm.chunk, filled = filled_chunks(n, chunks);
  if (c >= filled) return;
  uint32_t w0, w1;
  warp_units(n, filled, c, warp, &w0, &w1);
  const uint32_t lt = (1u << lane) - 1u;

  uint32_t cnt = 0;
  for (uint32_t u = w0; u < w1; ++u) {
    uint32_t k[kUnitRows];
#pragma unroll
    for (uint32_t j = 0; j < kUnitRows; ++j) {
      const uint32_t idx = u * kUnit + j * 32u + lane;
      k[j] = idx < n ? keys[idx] : kInvisibleKey;
    }
#pragma unroll
    for (uint32_t j = 0; j < kUnitRows; ++j) cnt += __popc(__ballot_sync(0xffffffffu, k[j] != kInvisibleKey));
  }
  if (lane == 0) sm.warp[warp] = cnt;
  uint32_t run, through;
  chunk_prefix(sm, status, c, ep.get(), ep.limit(), &ctl->error, &run, &through);
  if (c == filled - 1u && tid == 0) {
    ctl->visible_state[0] = through;
    ctl->visible_state[1] = through;
    ctl->visible_state[2] = (through + 1023u) / 1024u;
    ctl->visible_state[3] = 0u;
  }
  for (uint32_t u = w0; u < w1; ++u) {
    uint32_t k[kUnitRows];
#pragma unroll
    for (uint32_t j = 0; j < kUnitRows; ++j) {
      const uint32_t idx = u * kUnit + j * 32u + lane;
      k[j] = idx < n ? keys[idx] : kInvisibleKey;
    }
#pragma unroll
    for (uint32_t j = 0; j < kUnitRows; ++j) {
      const uint32_t idx = u * kUnit + j * 32u + lane;
      const bool vis = k[j] != kInvisibleKey;
      const uint32_t bal = __ballot_sync(0xffffffffu, vis);
      const uint32_t pos = run + __popc(bal & lt);
      if (idx < n) {
        vis_off[idx] = pos;
        if (vis) {
          keys_out[pos] = k[j];
          vals_out[pos] = idx;
        }
      }
      run += __popc(bal);
    }
  }
}

__global__ void __launch_bounds__(kBlock) k_frame_begin(uint32_t* base, uint32_t* __restrict__ zero,
                                                        uint32_t words) {
  for (uint32_t i = blockIdx.x * kBlock + threadIdx.x; i < words; i += gridDim.x * kBlock) zero[i] = 0u;
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  // Leaves room for kEpochsPerFrame launches; status words are 30-bit epochs.
  const uint32_t next = (*base + kEpochsPerFrame) & ((1u << 30) - 1u);
  *base = next < kEpochsPerFrame ? kEpochsPerFrame : next;
}

void launch_frame_begin(uint32_t* epoch_base, uint32_t* zero, uint32_t words, cudaStream_t st) {
  k_frame_begin<<<(words + kBlock * 4u - 1u) / (kBlock * 4u), kBlock, 0, st>>>(epoch_base, zero, words);
}

__global__ void k_skip_ticket(Control* ctl, uint32_t ticket) { ctl->tickets[ticket] += 1u; }

void launch_skip_ticket(Control* ctl, uint32_t ticket, cudaStream_t st) { k_skip_ticket<<<1, 1, 0, st>>>(ctl, ticket); }

uint32_t scan_chunks(uint32_t n_max, int sms) {
  const uint64_t units = ((uint64_t)n_max + kUnit - 1) / kUnit;
  return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(units, (uint64_t)kScanBlocksPerSm * (uint64_t)sms));
}

void launch_compact(const uint32_t* keys, uint32_t n, uint32_t* vis_off, uint32_t* keys_out, uint32_t* vals_out,
                    Control* ctl, unsigned long long* status, Epoch epoch, uint32_t chunks, cudaStream_t st) {
  k_compact<<<chunks, kBlock, 0, st>>>(keys, n, vis_off, keys_out, vals_out, ctl, status, epoch, chunks);
}

// Depth-ordered tile counts + saturating exclusive scan + prepare_dispatch +
// prepare_intersection_output (visibility.ts:63-76, scan.ts:9-99,
// intersections.ts:10-41,114-133) over the visible ranks. Phase 1 gathers
// each rank's tile count, writes it (the ordered counts) and reduces; phase 2
// re-reads the ordered counts and writes the saturating offsets.
__global__ void __launch_bounds__(kBlock) k_scan_counts(const uint32_t* __restrict__ ids,
                                                        const uint32_t* __restrict__ tile_counts,
                                                        uint32_t* __restrict__ ordered,
                                                        uint32_t* __restrict__ offsets, Control* __restrict__ ctl,
                                                        unsigned long long* __restrict__ status, Epoch ep,
                                                        uint32_t capacity, const uint32_t* __restrict__ frame_params,
                                                        uint32_t* __restrict__ output_state, uint32_t chunks) {
  __shared__ ScanShared sm;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (tid == 0) sm.chunk = atomicAdd(&ctl->tickets[kTicketScan], 1u);
  __syncthreads();
  const uint32_t n = ctl->visible_state[0];
  const uint32_t c = sm.chunk, filled = filled_chunks(n, chunks);
  if (c >= filled) return;
  uint32_t w0, w1;
  warp_units(n, filled, c, warp, &w0, &w1);

  uint32_t sum = 0;
  for (uint32_t u = w0; u < w1; ++u) {
    uint32_t id[kUnitRows];
#pragma unroll
    for (uint32_t j = 0; j < kUnitRows; ++j) {
      const uint32_t r = u * kUnit + j * 32u + lane;
      id[j] = r < n ? ids[r] : 0u;
    }
#pragma unroll
    for (uint32_t j = 0; j < kUnitRows; ++j) {
      const uint32_t r = u * kUnit + j * 32u + lane;
      if (r < n) {
        const uint32_t cnt = __ldg(tile_counts + id[j]);
        ordered[r] = cnt;
        sum = sat_add(sum, cnt);
      }
    }
  }
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) sum = sat_add(sum, __shfl_xor_sync(0xffffffffu, sum, d));
  if (lane == 0) sm.warp[warp] = sum;
  uint32_t run, all;
  chunk_prefix(sm, status, c, ep.get(), ep.limit(), &ctl->error, &run, &all);
  if (c == filled - 1u && tid == 0) {
    const bool overflow = all > capacity;
    const uint32_t count = overflow ? 0u : all;
    ctl->state[0] = count;
    ctl->state[1] = all;
    ctl->state[2] = (uint32_t)(((uint64_t)count + 1023u) / 1024u);
    ctl->state[3] = overflow ? 1u : 0u;
    const uint32_t attempt = frame_params[kFrameAttempt];
    const uint32_t last_version = frame_params[kFrameReset] ? 0u : output_state[1];
    output_state[0] = attempt;
    output_state[1] = overflow ? last_version : attempt;
    output_state[2] = all;
    output_state[3] = overflow ? 1u : 0u;
  }

  for (uint32_t u = w0; u < w1; ++u) {
    uint32_t cnt[kUnitRows];
#pragma unroll
    for (uint32_t j = 0; j < kUnitRows; ++j) {
      const uint32_t r = u * kUnit + j * 32u + lane;
      cnt[j] = r < n ? ordered[r] : 0u;  // written by this thread in phase 1
    }
#pragma unroll
    for (uint32_t j = 0; j < kUnitRows; ++j) {
      const uint32_t r = u * kUnit + j * 32u + lane;
      uint32_t incl = cnt[j];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= (uint32_t)d) incl = sat_add(y, incl);
      }
      const uint32_t excl = __shfl_up_sync(0xffffffffu, incl, 1);
      if (r < n) offsets[r] = sat_add(run, lane ? excl : 0u);
      run = sat_add(run, __shfl_sync(0xffffffffu, incl, 31));
    }
  }
}

void launch_scan_counts(const uint32_t* ids, const uint32_t* tile_counts, uint32_t* ordered, uint32_t* offsets,
                        Control* ctl, unsigned long long* status, Epoch epoch, uint32_t capacity,
                        const uint32_t* frame_params, uint32_t* output_state, uint32_t chunks, cudaStream_t st) {
  k_scan_counts<<<chunks, kBlock, 0, st>>>(ids, tile_counts, ordered, offsets, ctl, status, epoch, capacity,
                                           frame_params, output_state, chunks);
}

// ---------------------------------------------------------------------------
// Emission kernel (emit_group, emission.cuh).
// A block takes kBlock consecutive depth ranks. 5 blocks per SM (48
// registers): with no bound (60 registers, 4 blocks) 6M ranks took 206 us
// instead of 193, and two groups of ranks per block (64 registers; it paid
// off while the box rows were walked tile by tile) 1153 us instead of 1113 for
// 2 x 17.5M ranks.
template <bool PERIODIC>
__global__ void __launch_bounds__(kBlock, 5) k_emit(const uint32_t* __restrict__ ids, const float4* __restrict__ erec,
                                                    const uint32_t* __restrict__ ordered,
                                                    const uint32_t* __restrict__ offsets, BatchView bv, PassOptions o,
                                                    Control* __restrict__ ctl, uint32_t capacity,
                                                    uint32_t* __restrict__ tile_keys,
                                                    uint32_t* __restrict__ tile_vals) {
  if (ctl->state[3] != 0u) return;  // overflow: emission dispatch is zero
  __shared__ EmitShared sm;
  const uint32_t n = ctl->visible_state[0];
  const uint32_t first = blockIdx.x * kBlock;
  if (first >= n) return;  // whole block past the visible count
  const uint32_t r = first + threadIdx.x;
  uint32_t g = 0u, reserved = 0u, offset = 0u;
  float4 e0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), e1 = e0;
  if (r < n) {
    g = ids[r];
    reserved = ordered[r];
    offset = offsets[r];
    e0 = __ldg(erec + 2 * (size_t)g);
    e1 = __ldg(erec + 2 * (size_t)g + 1);
  }
  emit_group<PERIODIC>(sm, r < n, g, e0, e1, reserved, offset, bv, o, capacity, tile_keys, tile_vals);
}

void launch_emit(const uint32_t* ids, uint32_t n_max, const float4* erec, const uint32_t* ordered,
                 const uint32_t* offsets, const BatchView& b, const PassOptions& o, Control* ctl, uint32_t capacity,
                 uint32_t* tile_keys, uint32_t* tile_vals, cudaStream_t st) {
  if (n_max == 0) return;
  const uint32_t grid = (n_max - 1u) / kBlock + 1u;
  if (o.axis)
    k_emit<true><<<grid, kBlock, 0, st>>>(ids, erec, ordered, offsets, b, o, ctl, capacity, tile_keys, tile_vals);
  else
    k_emit<false><<<grid, kBlock, 0, st>>>(ids, erec, ordered, offsets, b, o, ctl, capacity, tile_keys, tile_vals);
}

// ---------------------------------------------------------------------------
// Tile ranges (tileOffsets.ts:4-128): offsets[t] = first sorted index with
// tile >= t, i.e. the reference's boundary detection followed by its
// suffix-min fill, written directly (offsets[T] = first sentinel or count).
__global__ void __launch_bounds__(kBlock) k_tile_ranges(const uint32_t* __restrict__ keys,
                                                        const Control* __restrict__ ctl, uint32_t ntile,
                                                        uint32_t* __restrict__ off) {
  // Each thread owns 8 consecutive boundaries i in [i0, i0 + 8), reading the
  // keys with two 16-byte loads (i0 is a multiple of 8).
  const uint32_t n = ctl->state[0];
  const uint32_t i0 = (blockIdx.x * kBlock + threadIdx.x) * 8u;
  if (i0 > n) return;
  uint32_t k[9];  // k[0] = keys[i0 - 1], k[1 + j] = keys[i0 + j]
  k[0] = i0 ? keys[i0 - 1] : 0u;
  if (i0 + 8u <= n) {
    const uint4 a = *reinterpret_cast<const uint4*>(keys + i0);
    const uint4 b = *reinterpret_cast<const uint4*>(keys + i0 + 4);
    k[1] = a.x; k[2] = a.y; k[3] = a.z; k[4] = a.w; k[5] = b.x; k[6] = b.y; k[7] = b.z; k[8] = b.w;
  } else {
#pragma unroll
    for (uint32_t j = 0; j < 8u; ++j) k[1 + j] = i0 + j < n ? keys[i0 + j] : 0u;
  }
#pragma unroll
  for (uint32_t j = 0; j < 8u; ++j) {
    const uint32_t i = i0 + j;
    if (i > n) break;
    const uint32_t lo = i == 0 ? 0u : k[j] + 1u;
    const uint32_t hi = i == n ? ntile : min(k[1 + j], ntile);
    for (uint32_t t = lo; t <= hi; ++t) off[t] = i;
  }
}

void launch_tile_ranges(const uint32_t* keys, Control* ctl, uint32_t ntile, uint32_t n_max, uint32_t* offsets,
                        cudaStream_t st) {
  const uint32_t grid = (uint32_t)(((uint64_t)n_max + 1 + 8ull * kBlock - 1) / (8ull * kBlock));
  k_tile_ranges<<<grid, kBlock, 0, st>>>(keys, ctl, ntile, offsets);
}

// ---------------------------------------------------------------------------
// Profiling diagnostics (ProfileDiagnosticsStage.ts:22-116).
//
// profileSubpixelCoverageWGSL (kernels/profileDiagnostics.ts:8-64): a
// projected splat counts when the projection marked it subpixel (mean.w < 0),
// or when its alpha-support box is at most one pixel in both dimensions and
// holds no pixel centre inside the support. Counted on the device instead of
// a per-splat flag buffer read back.
__global__ void __launch_bounds__(kBlock) k_zero_pixel(const float4* __restrict__ mean,
                                                       const float4* __restrict__ conic, BatchView bv,
                                                       uint32_t n, uint32_t* __restrict__ count) {
  const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
  uint32_t flag = 0;
  if (i < n) {
    const float4 m = mean[i];
    if (m.w < 0.0f) {
      flag = 1u;
    } else if (m.w > 0.0f) {
      const float4 c = conic[i];
      const float det = c.x * c.z - c.y * c.y;
      const float thr = gsdm::logf_(m.w * 255.0f);
      if (det > 1e-12f && thr > 0.0f) {
        const float s00 = c.z / det, s11 = c.x / det;
        const float ex = sqrtf(maxf((2.0f * thr) * s00, 0.0f)), ey = sqrtf(maxf((2.0f * thr) * s11, 0.0f));
        if (!(ex * 2.0f > 1.0f || ey * 2.0f > 1.0f)) {
          const ViewDesc& v = bv.views[find_view(bv.item_base, bv.nviews, i)];
          const int W = (int)v.vw, H = (int)v.vh;
          const int x0 = max((int)ceilf((m.x - ex) - 0.5f), 0), y0 = max((int)ceilf((m.y - ey) - 0.5f), 0);
          const int x1 = min((int)floorf((m.x + ex) - 0.5f), W - 1), y1 = min((int)floorf((m.y + ey) - 0.5f), H - 1);
          bool has = false;
          for (int py = y0; py <= y1; ++py)
            for (int px = x0; px <= x1; ++px) {
              const float dx = ((float)px + 0.5f) - m.x, dy = ((float)py + 0.5f) - m.y;
              const float sigma = 0.5f * ((c.x * dx * dx + 2.0f * c.y * dx * dy) + c.z * dy * dy);
              if (sigma <= thr) has = true;
            }
          flag = has ? 0u : 1u;
        }
      }
    }
  }
  const uint32_t warp_sum = __popc(__ballot_sync(0xffffffffu, flag != 0u));
  if ((threadIdx.x & 31u) == 0u && warp_sum) atomicAdd(count, warp_sum);
}

// Tile loads (utils/profileStats.ts:9-114): sums, maxima and threshold counts
// over offsets[t + 1] - offsets[t], the same for the loads capped at each of
// up to four caps, and a histogram of the loads (bin 65535 collects larger
// ones) from which the host reads the median and percentiles.
__global__ void __launch_bounds__(kBlock) k_tile_loads(const uint32_t* __restrict__ off, uint32_t ntile,
                                                       uint4 caps, TileLoadSums* __restrict__ out,
                                                       uint32_t* __restrict__ hist) {
  const uint32_t t = blockIdx.x * kBlock + threadIdx.x;
  if (t >= ntile) return;
  const uint32_t load = off[t + 1] > off[t] ? off[t + 1] - off[t] : 0u;
  atomicAdd(&out->total, (unsigned long long)load);
  atomicMax(&out->max, load);
  if (load > 256u) atomicAdd(&out->over[0], 1u);
  if (load > 512u) atomicAdd(&out->over[1], 1u);
  if (load > 1024u) atomicAdd(&out->over[2], 1u);
  if (load > 2048u) atomicAdd(&out->over[3], 1u);
  const uint32_t batches = (load + 255u) / 256u;
  atomicAdd(&out->batches, (unsigned long long)batches);
  atomicMax(&out->max_batches, batches);
  atomicAdd(&hist[min(load, 65535u)], 1u);
  const uint32_t cap[4] = {caps.x, caps.y, caps.z, caps.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (cap[k] == 0u) continue;
    const uint32_t r = min(load, cap[k]), d = load - r;
    atomicAdd(&out->cap_rasterized[k], (unsigned long long)r);
    if (d) {
      atomicAdd(&out->cap_dropped[k], (unsigned long long)d);
      atomicAdd(&out->cap_affected[k], 1u);
    }
    const uint32_t b = (r + 255u) / 256u;
    atomicAdd(&out->cap_batches[k], (unsigned long long)b);
    atomicMax(&out->cap_max_batches[k], b);
  }
}

void launch_profile(const float4* mean, const float4* conic, const BatchView& b, uint32_t n,
                    const uint32_t* tile_offsets, uint32_t ntile, const uint32_t caps[4], TileLoadSums* sums,
                    uint32_t* hist, uint32_t* zero_count, cudaStream_t st) {
  if (n) k_zero_pixel<<<(n + kBlock - 1) / kBlock, kBlock, 0, st>>>(mean, conic, b, n, zero_count);
  if (ntile)
    k_tile_loads<<<(ntile + kBlock - 1) / kBlock, kBlock, 0, st>>>(tile_offsets, ntile,
                                                                  make_uint4(caps[0], caps[1], caps[2], caps[3]),
                                                                  sums, hist);
}

// ---------------------------------------------------------------------------
void launch_raster_exact(const uint32_t* tile_offsets, const uint32_t* order, const uint32_t* ids,
                         const float4* mean, const float4* conic, const float4* color, const BatchView& b,
                         const PassOptions& o, Control* ctl, bool stats, cudaStream_t st) {
  launch_raster_policy<ExactMath>(tile_offsets, order, ids, mean, conic, color, b, o, ctl, stats, st);
}

}  // namespace gs
