// Visibility compaction that allocates nothing: gs3d_compact_visible_static.
//
// Who needs it: callers that cannot call cudaMalloc at the point where they
// enqueue work. A host that hands all device memory to its own arena or
// allocator (a game engine, a GPU process that manages memory on behalf of
// sandboxed clients) must not see allocations it did not make, and a
// real-time render loop must not stall on the driver's allocator, which may
// synchronise the device. Such callers pass their own input and output
// buffers; the kernel's scratch (the status words of the chunks, the
// per-call control block and the epoch counter) lives in the fixed
// device array below instead of memory allocated per pipeline.
//
// Cost of the array: kStaticScratchWords * 8 bytes (about 33 KB), held on
// every GPU that loads the library until the process exits.
//
// Rules for callers:
//  * The first call on a device resolves the array's device address with
//    cudaGetSymbolAddress (with that device current) and reads the device's
//    SM count; later calls skip that set-up. Each call enqueues two kernels on
//    the caller's stream: the compaction, and a one-block kernel that writes
//    `result` (count and error word).
//  * Every call on a device shares the one array. It starts as zeros, and each
//    call's last kernel zeroes the control block again; the status words
//    instead carry an epoch that the same kernel advances, so a previous
//    call's words never count as published (when the 30-bit epoch wraps, it
//    clears the words). A call whose second kernel could not be enqueued returns
//    GS3D_ERROR_CUDA, and the next call on the device clears the whole scratch
//    first. Calls that overlap on the GPU (two streams, or two host threads
//    without ordering) race on the array and give wrong results: order them
//    on one stream.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "../../include/gs3d.h"
#include "pass_common.cuh"

using namespace gs;

namespace {

constexpr size_t kControlWords = (sizeof(Control) + 7) / 8;
constexpr size_t kStatusWords = 4096;  // one per chunk of k_compact; the grid is capped to this
constexpr size_t kEpochWords = 1;      // the epoch counter (low 32 bits of the word)
constexpr size_t kStaticScratchWords = kControlWords + kStatusWords + kEpochWords;
static_assert(sizeof(Control) % 8 == 0, "control block must be a whole number of words");

// The scratch: control block, status words, epoch counter.
static __device__ __align__(256) unsigned long long g_compact_scratch[kStaticScratchWords];

constexpr int kMaxDevices = 64;
std::mutex g_mutex;
unsigned long long* g_scratch_ptr[kMaxDevices] = {};
int g_sms[kMaxDevices] = {};
bool g_unfinished[kMaxDevices] = {};  // a call's compaction went out without its last kernel
std::atomic<bool> g_refuse_finish{false};

// Hands the results out and leaves the scratch ready for the next call: the
// control block zeroed, the epoch counter advanced by one (when the 30-bit
// counter wraps, with every status word cleared, so that no word left by an
// earlier call can carry a later one's epoch). Bound by its launch; a kernel
// that advanced the epoch, a memset and two copies took four: 1000 keys 23.2
// -> 13.0 us, 100k 32.5 -> 20.1, 5M 40.6 -> 30.3 (with the chunks' sums; 27 with
// overlapped launches).
__global__ void __launch_bounds__(256) k_static_finish(Control* ctl, unsigned long long* status, uint32_t* epoch,
                                                       unsigned char* result) {
  after_previous();
  const uint32_t tid = threadIdx.x;
  // By bytes: the words of `result` may lie at any address.
  if (tid < 8u) {
    const uint32_t word = tid < 4u ? ctl->visible_state[0] : ctl->error;
    result[tid] = (unsigned char)(word >> (8u * (tid & 3u)));
  }
  const uint32_t next = *epoch + 1u;
  __syncthreads();  // every thread has read the control block and the counter
  const bool wrap = next >= (1u << 30) - 1u;
  for (uint32_t i = tid; i < kControlWords; i += blockDim.x) reinterpret_cast<unsigned long long*>(ctl)[i] = 0ull;
  if (wrap)
    for (uint32_t i = tid; i < kStatusWords; i += blockDim.x) status[i] = 0ull;
  if (tid == 0) *epoch = wrap ? 0u : next;
}

}  // namespace

extern "C" gs3d_status gs3d_compact_visible_static(const uint32_t* keys, uint32_t n, uint32_t* visible_offsets,
                                                   uint32_t* keys_out, uint32_t* ids_out, uint32_t* result,
                                                   void* stream) {
  if (n > GS3D_STATIC_COMPACT_MAX_ITEMS) return GS3D_ERROR_RANGE;
  if (!result || (n > 0 && (!keys || !visible_offsets || !keys_out || !ids_out)))
    return GS3D_ERROR_INVALID_ARGUMENT;
  if (((uintptr_t)keys & 3u) != 0) return GS3D_ERROR_INVALID_ARGUMENT;  // read as 4-byte words
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDevices) return GS3D_ERROR_CUDA;
  cudaStream_t st = (cudaStream_t)stream;
  unsigned long long* scratch = nullptr;
  int sms = 1;
  bool clear = false;
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_scratch_ptr[device]) {
      // One-time set-up on this device (the current device).
      void* p = nullptr;
      if (cudaGetSymbolAddress(&p, g_compact_scratch) != cudaSuccess || !p) {
        cudaGetLastError();
        return GS3D_ERROR_CUDA;
      }
      if (cudaDeviceGetAttribute(&g_sms[device], cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        cudaGetLastError();
        return GS3D_ERROR_CUDA;
      }
      g_scratch_ptr[device] = (unsigned long long*)p;
    }
    scratch = g_scratch_ptr[device];
    sms = g_sms[device];
    clear = g_unfinished[device];
  }
  Control* ctl = reinterpret_cast<Control*>(scratch);
  unsigned long long* status = scratch + kControlWords;
  uint32_t* epoch = reinterpret_cast<uint32_t*>(scratch + kControlWords + kStatusWords);
  if (clear) {
    // The tickets of a compaction that no last kernel followed are used up and
    // its sums carry the epoch of this call: start again from zeros. A call
    // that is only being captured leaves that to the next one as well.
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &capture) != cudaSuccess ||
        cudaMemsetAsync(scratch, 0, kStaticScratchWords * sizeof(unsigned long long), st) != cudaSuccess) {
      cudaGetLastError();
      return GS3D_ERROR_CUDA;
    }
    std::lock_guard<std::mutex> lock(g_mutex);
    if (capture == cudaStreamCaptureStatusNone) g_unfinished[device] = false;
  }
  const uint32_t chunks = std::min<uint32_t>(scan_chunks(n, sms), (uint32_t)kStatusWords);
  launch_compact(keys, n, visible_offsets, keys_out, ids_out, ctl, status, Epoch{epoch, 1u, 0u}, chunks, st);
  cudaError_t finish = cudaErrorLaunchOutOfResources;
  if (!g_refuse_finish.exchange(false))
    finish = launch_after(k_static_finish, 1, 256, 0, st, ctl, status, epoch, (unsigned char*)result);
  if (finish != cudaSuccess) {
    cudaGetLastError();
    std::lock_guard<std::mutex> lock(g_mutex);
    g_unfinished[device] = true;
    return GS3D_ERROR_CUDA;
  }
  if (cudaGetLastError() != cudaSuccess) return GS3D_ERROR_CUDA;
  return GS3D_OK;
}

extern "C" void gs3d_debug_refuse_compact_finish(void) { g_refuse_finish.store(true); }
