// Shared definitions of the CUDA pass: kernel parameter blocks, the per-frame
// control block, and the status words by which the chunks of the compaction
// and scan kernels tell each other their sums.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace gs {

constexpr int kBlock = 256;  // threads per block for the linear kernels
constexpr uint32_t kTileSize = 16;  // the reference's pixels per tile side (src/renderer/pipeline/constants.ts:1)

// One view of a batch: a scene (packed GaussianData buffers), a camera
// (FrameUniforms.ts:18-58 + the object table), a viewport and its targets.
// Views are concatenated: view v owns items [item_base, item_base + active)
// (item_base is a multiple of kBlock so every projection block belongs to one
// view) and global tile ids [tile_base, tile_base + tiles_x * tiles_y).
struct ViewDesc {
  const float4* means;     // count
  const uint2* shape;      // count
  const uint32_t* rot;     // count
  const uint32_t* sh;      // count * C + count (active tail at count * C)
  const float* objects;    // object_count * 40
  void* color;             // rgba16f or rgba32f, width * height
  float* depth;            // width * height or null
  uint32_t count, active, degree, C;
  uint32_t object_count, color_half;
  uint32_t tiles_x, tiles_y;
  uint32_t item_base, tile_base, pad0, pad1;
  float P[16];             // projection, column-major
  float vw, vh, vnear, vfar;
};

// Pass options shared by every view (TiledGaussianPipeline constructor options).
struct PassOptions {
  float filter;
  uint32_t axis;           // boundary axis 0/1/2
  uint32_t antialias;      // 0 compensated, 1 classic
  uint32_t subpixel;       // subpixel sample culling
  uint32_t depth_mode;     // 0 float32, 1 packed16
  uint32_t chunk;          // raster chunk size, 0 = none
  uint32_t max_per_tile;   // 0 = uncapped
  uint32_t depth_encoding; // 0 device depth, 1 raw
  float background[4];
  float t_threshold;
  float depth_alpha_threshold;
  float invalid_depth;
  uint32_t proj_fp64;      // 1: FP64 far-origin mean transform and near-singular conic
  uint32_t any_depth;      // some view of the launch has a depth target
  uint32_t tile;           // pixels per tile side: 16 (the reference's), or 8 / 32 in tuned batches
  float tile_px;           // the same as a float
  float tile_inv;          // its reciprocal (exact: a power of two)
  uint32_t pixels_per_lane;  // fast raster forms: 2 (a warp per 8x8 patch) or 4 (per 8x16)
};

// The per-frame parameters at the head of a staged batch table. All but the
// first two are the fused front's (front.cu), at their start values with every
// copy: the range of the visible depth keys and the counters of its barriers,
// each on an L2 line of its own (they are polled).
enum FrameParam : uint32_t {
  kFrameAttempt = 0,
  kFrameReset = 1,
  kFrameKeyMin = 2,
  kFrameKeyMax = 3,
  kFrameBarrier = 32,
  kFrameDepthBarrier = 64,
  kFrameTileBarrier = 96,
  kFrameParams = 128
};

// The batch table in device memory: the per-frame parameters
// (FrameParam), four ascending arrays (nviews + 1 entries each), then the view
// descriptors. Consecutive views that render the same packed scene form a view
// group, projected together (group_block: first projection block of each
// group; group_view: first view of each group; ngroups + 1 entries used).
struct BatchView {
  const uint32_t* item_base;
  const uint32_t* tile_base;
  const uint32_t* group_block;
  const uint32_t* group_view;
  const ViewDesc* views;
  const uint32_t* frame_params;  // FrameParam
  uint32_t nviews;
  uint32_t ngroups;
  uint32_t total_items;
  uint32_t total_tiles;
  uint32_t total_blocks;         // projection blocks over the groups
};

// Index of the view whose [base[v], base[v+1]) range holds x.
__device__ __forceinline__ uint32_t find_view(const uint32_t* base, uint32_t nviews, uint32_t x) {
  uint32_t lo = 0, hi = nviews;  // base[lo] <= x < base[hi]
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(base + mid) <= x) lo = mid; else hi = mid;
  }
  return lo;
}

// Overlapped launches: a kernel launched by launch_after starts with a wait
// for all of the kernel before it on the stream, its writes included
// (after_previous), so that its launch is out of the way when that one ends;
// if the kernel before says next_may_launch, its blocks also move in where
// that one's last blocks leave. Used where the next kernel's blocks are as
// many per SM as fit (the scatter after the count: 3) or come in many waves
// (the rasterizer): 3M splats at 1080p 909 -> 896 us, 6M at 1440p 1346 -> 1335,
// eight objects 3604 -> 3578, compaction of 1000 keys 13.0 -> 9.9. A
// persistent kernel with room for more blocks per SM than its grid has (count,
// compaction, scan) moves in unevenly and then runs as long as its fullest SM
// (depth sort of 6M 178 -> 198 us), and the wait costs the projection and the
// emission, of tens of waves, more than it saves (48M ordinals: +2%).
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void next_may_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launches a kernel that begins with after_previous().
template <typename... P, typename... A>
cudaError_t launch_after(void (*kernel)(P...), uint32_t grid, uint32_t block, size_t dynamic, cudaStream_t st, A... args) {
  cudaLaunchAttribute overlap = {};
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(grid);
  config.blockDim = dim3(block);
  config.dynamicSmemBytes = dynamic;
  config.stream = st;
  config.attrs = &overlap;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, kernel, static_cast<P>(args)...);
}

constexpr uint32_t kMaxSortPasses = 4;  // passes of a tile sort
// Persistent blocks per SM of the chunked scans (compaction and
// ordered-count scan); scan_chunks() = their grid for n_max items.
constexpr uint32_t kScanBlocksPerSm = 4;
uint32_t scan_chunks(uint32_t n_max, int sms);

// Per-frame control block, zeroed before each render.
struct Control {
  uint32_t tickets[2];           // dynamic chunk ids of the chunked scans (Ticket)
  uint32_t visible_state[4];     // visible, visible, radix blocks, 0
  uint32_t state[4];             // count, total, radix blocks, overflow
  uint32_t error;                // ErrorBit
  uint32_t pad[3];
  unsigned long long raster_stats[4];  // checked, blended, pixels, alpha-stopped
  uint32_t order_hist[34];       // raster work-list buckets (tile load classes)
  uint32_t order_fill[34];
};

enum ErrorBit : uint32_t {
  kErrorWait = 1u,  // a chunk-sum wait or a grid barrier expired
  kErrorCopy = 4u   // a sort tile's copy never landed
};

enum Ticket { kTicketCompact = 0, kTicketScan = 1 };

// ---------------------------------------------------------------------------
// Status words of the chunked scans: [63:32] epoch, [31:0] the chunk's sum.
// A word whose epoch differs from the launch's epoch is "not yet published",
// so the status array never needs clearing between launches. A frame's
// launches use epochs base + 1 .. base + kEpochsPerFrame, where base is a
// device-side counter advanced by k_frame_begin at the start of every frame,
// so a replayed CUDA graph never reuses an epoch.
constexpr uint32_t kEpochsPerFrame = 16;

constexpr uint32_t kSpinLimit = 1u << 22;  // default polls before a wait is declared expired (one to a few seconds)

// The epoch of chunked-scan launch `add` of the current frame, and how many
// polls a wait of that launch may spend on one status word.
struct Epoch {
  const uint32_t* base;  // device counter
  uint32_t add;
  uint32_t spin_limit;   // 0: kSpinLimit
  __device__ __forceinline__ uint32_t get() const { return *base + add; }
  __device__ __forceinline__ uint32_t limit() const { return spin_limit ? spin_limit : kSpinLimit; }
};

// A status word carries its value, so no other memory hangs on its order.
__device__ __forceinline__ unsigned long long ld_status(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_status(unsigned long long* p, uint32_t epoch, uint32_t value) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(((unsigned long long)epoch << 32) | value)
               : "memory");
}
__device__ __forceinline__ uint32_t sat_add(uint32_t a, uint32_t b) { return a + min(b, 0xffffffffu - a); }

// Wait (bounded) until *p, last read as v, carries this launch's epoch; its
// value. On expiry the error word gets kErrorWait and the value is zero, so the
// kernel always finishes and the host sees the error.
__device__ __forceinline__ uint32_t wait_status(const unsigned long long* p, unsigned long long v, uint32_t epoch,
                                                uint32_t limit, uint32_t* err) {
  uint32_t polls = 0, backoff = 8;
  while ((uint32_t)(v >> 32) != epoch) {
    if (++polls >= limit) {
      atomicOr(err, kErrorWait);
      return 0;
    }
    __nanosleep(backoff);
    backoff = backoff < 256 ? backoff * 2 : 256;
    v = ld_status(p);
  }
  return (uint32_t)v;
}

// ---------------------------------------------------------------------------
// Block-wide exclusive scan of one value per thread (256 threads).
template <bool SATURATE>
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* s_warp, uint32_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x = SATURATE ? sat_add(y, x) : y + x;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < (kBlock / 32) ? s_warp[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w = SATURATE ? sat_add(y, w) : y + w;
    }
    if (lane < (kBlock / 32)) s_warp[lane] = w;
  }
  __syncthreads();
  uint32_t warp_prefix = warp == 0 ? 0u : s_warp[warp - 1];
  uint32_t incl = SATURATE ? sat_add(warp_prefix, x) : warp_prefix + x;
  *total = s_warp[kBlock / 32 - 1];
  // Exclusive value = the previous thread's inclusive value (exact for the
  // saturating form too, since saturating addition is associative).
  uint32_t prev = __shfl_up_sync(0xffffffffu, incl, 1);
  uint32_t excl = lane == 0 ? warp_prefix : prev;
  __syncthreads();
  return excl;
}

constexpr uint32_t kProjectBlocksPerSm = 4;  // resident blocks of the projection kernel

// Launch wrappers implemented in the .cu files.
// Packed raster record of a visible splat, read by the fast raster forms with
// one 32-byte gather (two float4, 32-byte aligned):
//   [0] cx, cy, -a/2 log2 e, -b log2 e
//   [1] -c/2 log2 e, log2 opacity, half2(r, g) bits, half2(b, min(log2 opacity, log2 0.99)) bits
// where (a, b, c) is the conic. Written by the projection when `rec` is not null.
// rec: packed raster records of the fast forms (null for EXACT); erec: the
// emission records, two float4 per item: (cx, cy, conic a, conic b),
// (conic c, log(opacity * 255), rx + 512 ry, 1 if the box has to be walked tile
// by tile, else 0), written for visible items.
void launch_project(const BatchView& b, const PassOptions& o, float4* mean, float4* conic, float4* color,
                    uint32_t* counts, uint32_t* keys, float4* rec, float4* erec, cudaStream_t st);
// Starts a frame: advances the epoch of the status words and clears `words` words (the
// sorts' sums and the control block).
void launch_frame_begin(uint32_t* epoch_base, uint32_t* zero, uint32_t words, cudaStream_t st);
// Advance ticket counter `ticket` of the control block by one (a test hook:
// the chunk of ticket 0 is then never scanned, so the waits for its
// sum run out).
void launch_skip_ticket(Control* ctl, uint32_t ticket, cudaStream_t st);
void launch_compact(const uint32_t* keys, uint32_t n, uint32_t* vis_off, uint32_t* keys_out, uint32_t* vals_out,
                    Control* ctl, unsigned long long* status, Epoch epoch, uint32_t chunks, cudaStream_t st);
void launch_scan_counts(const uint32_t* sorted_ids, const uint32_t* tile_counts, uint32_t* ordered,
                        uint32_t* offsets, Control* ctl, unsigned long long* status, Epoch epoch,
                        uint32_t capacity, const uint32_t* frame_params, uint32_t* output_state, uint32_t chunks,
                        cudaStream_t st);
void launch_emit(const uint32_t* sorted_ids, uint32_t n_max, const float4* erec, const uint32_t* ordered,
                 const uint32_t* offsets, const BatchView& b, const PassOptions& o, Control* ctl, uint32_t capacity,
                 uint32_t* tile_keys, uint32_t* tile_vals, cudaStream_t st);
void launch_tile_ranges(const uint32_t* sorted_tile_keys, Control* ctl, uint32_t ntile, uint32_t n_max,
                        uint32_t* tile_offsets, cudaStream_t st);
constexpr uint32_t kSortTile = 4096;  // items per sort tile
// Chunked LSD pass (reduce, scatter; no look-back chain) over the digit of
// `bits` bits from `shift` on of the key, or, at 9 bits (the most), of
// key - low: `chunks` blocks, each walking a contiguous run of 4096-item tiles. counts holds chunks rows
// of 2^bits words; sums (sum_rows(chunks) rows of kSumWords words, zero on
// entry) takes the counts of 16 chunks a row; spare, as large, is zeroed (the
// next pass takes it as its sums). n is read from *n_ptr on the device.
constexpr uint32_t kChunkBlocksPerSm = 3;
constexpr uint32_t kSumChunks = 16;
constexpr uint32_t kSumWords = 512;
__host__ __device__ constexpr uint32_t sum_rows(uint32_t chunks) { return (chunks + kSumChunks - 1u) / kSumChunks; }
uint32_t chunk_pass_chunks(uint32_t n_max, int sms);
// err: the control block's error word (kErrorCopy).
void launch_chunk_pass(int bits, const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out,
                       uint32_t* vals_out, const uint32_t* n_ptr, uint32_t low, int shift, uint32_t chunks,
                       uint32_t* counts, uint32_t* sums, uint32_t* spare, uint32_t* err, cudaStream_t st);
// Opt every sort-scatter instantiation into its shared-memory size (once per
// device; call before any stream capture).
void prepare_sort_kernels();
// The fused front of small launches (front.cu): the stages before the
// rasterizer in one cooperative kernel of kFrontBlocksPerSm blocks per SM at
// most. front_fits: whether the (current) device takes cooperative launches
// and holds all of these blocks at once. frame_params: the staged
// table's FrameParam words on the device. tile_order null: no work list.
// wait_limit: polls of a barrier (0: kSpinLimit). withhold: block 0 leaves before
// the compaction (a test hook: the others' next barrier expires).
// launch_front's status: on an error nothing was enqueued (a stream or a
// context that may use only some of the device's SMs can refuse the launch).
constexpr uint32_t kFrontBlocksPerSm = 3;
size_t front_scratch_words(int sms);  // words of FrontBuffers::scratch
struct FrontBuffers {
  float4 *mean, *conic, *color, *rec, *erec;
  uint32_t *tile_counts, *keys, *vis_off, *dk[2], *dv[2], *ordered, *ioff, *tk[2], *tv[2];
  uint32_t *tile_offsets, *tile_order, *scratch;
  Control* ctl;
  uint32_t* output_state;
};
bool front_fits(int device);
cudaError_t launch_front(const BatchView& b, const PassOptions& o, const FrontBuffers& w, uint32_t* frame_params,
                         uint32_t capacity, uint32_t tile_passes, uint32_t digit_bits, int sms, uint32_t wait_limit,
                         bool withhold, cudaStream_t st);
// Raster work list: every tile of the batch, heaviest load class first.
void launch_tile_order(const uint32_t* tile_offsets, uint32_t ntile, Control* ctl, uint32_t* order, int sms,
                       cudaStream_t st);
// Rasterizer over every tile of the batch (precision: 0 fp32, 1 exact, 2 half2).
void launch_raster(int precision, const uint32_t* tile_offsets, const uint32_t* order, const uint32_t* sorted_ids,
                   const float4* mean, const float4* conic, const float4* color, const float4* rec,
                   const BatchView& b, const PassOptions& o, Control* ctl, bool stats, cudaStream_t st);
// Profiling diagnostics: tile-load sums (caps: up to four, 0 = unused) and
// the zero-pixel subpixel splat count (ProfileDiagnosticsStage.ts:22-116).
struct TileLoadSums {
  unsigned long long total, batches;
  uint32_t max, max_batches, over[4];
  unsigned long long cap_rasterized[4], cap_dropped[4], cap_batches[4];
  uint32_t cap_affected[4], cap_max_batches[4];
};
void launch_profile(const float4* mean, const float4* conic, const BatchView& b, uint32_t n,
                    const uint32_t* tile_offsets, uint32_t ntile, const uint32_t caps[4], TileLoadSums* sums,
                    uint32_t* hist, uint32_t* zero_count, cudaStream_t st);
void launch_raster_exact(const uint32_t* tile_offsets, const uint32_t* order, const uint32_t* sorted_ids,
                         const float4* mean, const float4* conic, const float4* color, const BatchView& b,
                         const PassOptions& o, Control* ctl, bool stats, cudaStream_t st);

}  // namespace gs
