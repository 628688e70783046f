// On-device compact packer: linear splat attributes -> the packed storage
// buffers the pass consumes (GaussianData.ts:10-33).
// Restates, on the GPU, the reference's CPU packer for the compact layout:
//   rust/gaussian-backend/src/engine.rs:1801-1891 encode_attributes (compact):
//     means          (x, y, z, objectId)
//     scalesOpacity  [f16 ln sx | f16 ln sy << 16, f16 ln sz | f16 opacity << 16]
//                    (rust/vendor/spark-lib/src/splat_encode.rs:127-136 encode_ext_splat)
//     rotations      oct101012 of the normalised quaternion (splat_encode.rs:234-252)
//     shCoefficients rgb8e8 words: DC = (rgb - 0.5) / SH_C0, then the higher bands
//                    (engine.rs:1857-1872, pack_sh :1940-1949)
// Built with --fmad=false so products and sums round like the Rust code.
// f16 conversion rounds to nearest even (half::f16::from_f32), round() is half
// away from zero (f32::round), the rgb8e8 exponent is ceil(log2 max|c|)
// computed exactly from the binary exponent. ln, acos and sin are CUDA's; where
// a result sits within an ulp of a quantisation boundary the packed field can
// differ by one step from the CPU packer's.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/gs3d.h"

namespace {

constexpr float kShC0 = 0.28209479177387814f;  // engine.rs:1858
constexpr float kPi = 3.14159265358979323846f;

__device__ __forceinline__ uint32_t f16_bits(float x) { return (uint32_t)__half_as_ushort(__float2half_rn(x)); }

__device__ __forceinline__ float clampf(float v, float lo, float hi) { return v < lo ? lo : (v > hi ? hi : v); }

// splat_encode.rs:234-252 encode_quat_oct101012.
__device__ uint32_t encode_oct101012(float qx, float qy, float qz, float qw) {
  if (qw < 0.0f) {
    qx = -qx; qy = -qy; qz = -qz; qw = -qw;
  }
  const float theta = 2.0f * acosf(clampf(qw, 0.0f, 1.0f));
  const float s = sinf(theta * 0.5f);
  float ax = 1.0f, ay = 0.0f, az = 0.0f;
  if (!(fabsf(s) < 1e-6f)) {
    ax = qx / s; ay = qy / s; az = qz / s;
  }
  const float sum = (fabsf(ax) + fabsf(ay)) + fabsf(az);
  float p0 = ax / sum, p1 = ay / sum;
  if (az < 0.0f) {
    const float f0 = (1.0f - fabsf(p1)) * (p0 >= 0.0f ? 1.0f : -1.0f);
    const float f1 = (1.0f - fabsf(p0)) * (p1 >= 0.0f ? 1.0f : -1.0f);
    p0 = f0; p1 = f1;
  }
  const uint32_t u = (uint32_t)roundf(clampf((p0 * 0.5f + 0.5f) * 1023.0f, 0.0f, 1023.0f));
  const uint32_t v = (uint32_t)roundf(clampf((p1 * 0.5f + 0.5f) * 1023.0f, 0.0f, 1023.0f));
  const uint32_t r = (uint32_t)roundf(clampf(theta / kPi * 4095.0f, 0.0f, 4095.0f));
  return (r << 20) | (v << 10) | u;
}

// The shared exponent of engine.rs:1945, `max.log2().ceil()` on an f32: the
// ceiling of log2 rounded to f32. It equals the exact ceiling except just
// above a power of two 2^e (e != 0), where log2 rounds down to e itself and
// the exponent stays e instead of e + 1. Decided exactly: the f32 neighbour
// of e towards e + 1 lies ulp(e) above a positive e, and below |e| by
// ulp(|e|) (half that when |e| is a power of two) for a negative e; log2
// rounds to e when log2(m) is under half that gap, h = 2^(g - 1). With the
// mantissa m = 1 + j 2^-23 that is j < 2^23 (2^h - 1) = 2^(g + 22) ln 2 plus
// a term below 2e-4 (h <= 2^-17), and no 2^(g + 22) ln 2 with g in [-24, -16]
// lies that close below an integer, so j is compared with the product in
// FP32 (this was a double log1p per SH word, 16 per splat: the whole kernel
// ran at the FP64 rate). mx > 0 and not subnormal results below -126 are
// clamped by the caller.
__device__ __forceinline__ int rounded_log2_ceil(float mx) {
  const uint32_t b = __float_as_uint(mx);
  const int field = (int)(b >> 23);
  const uint32_t j = b & 0x7fffffu;
  if (field == 255) return j ? 0 : 127;  // NaN: Rust's saturating cast; infinity is clamped to 127
  if (field == 0) return -126;           // subnormal: at most -126 before the clamp
  const int e = field - 127;
  if (j == 0u) return e;                 // a power of two
  if (e == 0) return 1;                  // log2 m itself is representable: above 0
  const int a = e > 0 ? e : -e;
  const int g = (31 - __clz(a)) - 23 - (e < 0 && (a & (a - 1)) == 0 ? 1 : 0);
  const float limit = __uint_as_float(0x3f317218u + ((uint32_t)(g + 22) << 23));  // 2^(g + 22) ln 2
  return (float)j < limit ? e : e + 1;
}

// engine.rs:1940-1949 pack_sh.
__device__ __forceinline__ uint32_t pack_sh(float r, float g, float b) {
  const float mx = fmaxf(fmaxf(fabsf(r), fabsf(g)), fabsf(b));
  if (mx == 0.0f) return 0u;
  int e = rounded_log2_ceil(mx);
  e = e < -126 ? -126 : (e > 127 ? 127 : e);
  // 127 / 2^e: exact, 127 = 1.984375 2^6 with the exponent moved by -e, or
  // infinity past the largest float.
  const float mult = __uint_as_float(e < -121 ? 0x7f800000u : ((uint32_t)(133 - e) << 23) | 0x7e0000u);
  const float c[3] = {r, g, b};
  uint32_t w = (uint32_t)(e + 127) << 24;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float q = clampf(floorf(c[i] * mult + 0.5f), -127.0f, 127.0f);
    w |= ((uint32_t)(int32_t)q & 255u) << (8 * i);
  }
  return w;
}

constexpr uint32_t kPackBlock = 256;  // splats, and threads, of a block

// HBM-bound: 4 (14 + 3 (C - 1)) bytes read and 28 + 4 C written per splat. A
// block takes 256 consecutive splats: one thread per splat for the geometry
// and the colour's word, then its 256 C SH words spread over the threads, so
// that the coefficient reads (12 consecutive bytes per thread) and the word
// stores of a warp are consecutive; with a thread per splat they lay C words
// apart. The colour's word comes through shared memory: computed in the loop,
// its three divisions ran in nearly every warp for two of 32 lanes. Four words
// of a thread are in flight (2 and 8: 56 and 70 us against 60 at degree 2, 76
// and 81 against 76 at degree 3).
// 1M splats at degree 3: 1810 us with a thread per splat and the double
// log1p, 90 us with the words spread, 72 us (4.6 TB/s) so; 4M 322 and 261 us.
template <uint32_t C>
__global__ void __launch_bounds__(kPackBlock) k_pack(gs3d_splat_source src, uint32_t first,
                                                     float4* __restrict__ means, uint2* __restrict__ shape,
                                                     uint32_t* __restrict__ rot, uint32_t* __restrict__ sh) {
  __shared__ uint32_t s_colour[kPackBlock];  // first SH words: the colours
  const uint32_t i0 = blockIdx.x * kPackBlock;
  const uint32_t count = min(kPackBlock, src.count - i0);
  if (threadIdx.x < count) {
    const uint32_t i = i0 + threadIdx.x;
    const size_t slot = (size_t)first + i;
    const float cx = src.centers[3 * (size_t)i], cy = src.centers[3 * (size_t)i + 1], cz = src.centers[3 * (size_t)i + 2];
    means[slot] = make_float4(cx, cy, cz, (float)src.object_id);
    const float sx = src.scales[3 * (size_t)i], sy = src.scales[3 * (size_t)i + 1], sz = src.scales[3 * (size_t)i + 2];
    shape[slot] = make_uint2(f16_bits(logf(sx)) | (f16_bits(logf(sy)) << 16),
                             f16_bits(logf(sz)) | (f16_bits(src.opacity[i]) << 16));
    // glam Quat::normalize: multiply by the reciprocal of the length.
    const float* q = src.quaternions + 4 * (size_t)i;
    const float inv = 1.0f / sqrtf(((q[0] * q[0] + q[1] * q[1]) + q[2] * q[2]) + q[3] * q[3]);
    rot[slot] = encode_oct101012(q[0] * inv, q[1] * inv, q[2] * inv, q[3] * inv);
    const float* rgb = src.rgb + 3 * (size_t)i;
    s_colour[threadIdx.x] =
        pack_sh((rgb[0] - 0.5f) / kShC0, (rgb[1] - 0.5f) / kShC0, (rgb[2] - 0.5f) / kShC0);
  }
  __syncthreads();
  uint32_t* out = sh + ((size_t)first + i0) * C;
  const float* rest = src.sh_rest + (size_t)i0 * (C - 1u) * 3u;
  constexpr uint32_t kAtOnce = C < 4u ? C : 4u;  // words of a thread in flight
  for (uint32_t w0 = threadIdx.x; w0 < count * C; w0 += kAtOnce * kPackBlock) {
    float c[kAtOnce][3];
#pragma unroll
    for (uint32_t j = 0; j < kAtOnce; ++j) {
      const uint32_t w = w0 + j * kPackBlock, i = w / C;
      const bool read = w < count * C && w != i * C;
      const float* at = rest + (w - i - 1u) * 3u;  // word k of splat i: i (C - 1) + k - 1 coefficients precede it
      c[j][0] = read ? at[0] : 0.0f;
      c[j][1] = read ? at[1] : 0.0f;
      c[j][2] = read ? at[2] : 0.0f;
    }
#pragma unroll
    for (uint32_t j = 0; j < kAtOnce; ++j) {
      const uint32_t w = w0 + j * kPackBlock, i = w / C;
      if (w < count * C) out[w] = w == i * C ? s_colour[i] : pack_sh(c[j][0], c[j][1], c[j][2]);
    }
  }
}

}  // namespace

extern "C" gs3d_status gs3d_pack_splats(const gs3d_splat_source* src, uint32_t first_slot, float* means,
                                        uint32_t* scales_opacity, uint32_t* rotations, uint32_t* sh_coefficients,
                                        uint32_t capacity, void* stream) {
  if (!src || !means || !scales_opacity || !rotations || !sh_coefficients) return GS3D_ERROR_INVALID_ARGUMENT;
  if (src->sh_degree > 3) return GS3D_ERROR_RANGE;
  if ((uint64_t)first_slot + src->count > capacity) return GS3D_ERROR_RANGE;
  if (src->count == 0) return GS3D_OK;
  if (!src->centers || !src->scales || !src->opacity || !src->quaternions || !src->rgb ||
      (src->sh_degree > 0 && !src->sh_rest))
    return GS3D_ERROR_INVALID_ARGUMENT;
  if (((uintptr_t)means & 15u) || ((uintptr_t)scales_opacity & 7u)) return GS3D_ERROR_INVALID_ARGUMENT;
  const uint32_t grid = (src->count - 1u) / kPackBlock + 1u;
  cudaStream_t st = (cudaStream_t)stream;
  float4* m = reinterpret_cast<float4*>(means);
  uint2* s = reinterpret_cast<uint2*>(scales_opacity);
  switch (src->sh_degree) {
    case 0: k_pack<1><<<grid, kPackBlock, 0, st>>>(*src, first_slot, m, s, rotations, sh_coefficients); break;
    case 1: k_pack<4><<<grid, kPackBlock, 0, st>>>(*src, first_slot, m, s, rotations, sh_coefficients); break;
    case 2: k_pack<9><<<grid, kPackBlock, 0, st>>>(*src, first_slot, m, s, rotations, sh_coefficients); break;
    default: k_pack<16><<<grid, kPackBlock, 0, st>>>(*src, first_slot, m, s, rotations, sh_coefficients); break;
  }
  return cudaGetLastError() == cudaSuccess ? GS3D_OK : GS3D_ERROR_CUDA;
}
