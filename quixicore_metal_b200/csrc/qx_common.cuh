// Shared host/device helpers for the B200 backend: element-type conversion, the epilogue math,
// the stateless RNG hash and the status / launch bookkeeping used by every translation unit.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/quixicore_cuda.h"

namespace qx {

// ---- launch bookkeeping -------------------------------------------------------------------
void note_launch(int n = 1);                       // counts kernels this library enqueued
qx_status ok(const char* op);
qx_status fail(qx_status_code code, const char* op, const char* detail);
qx_status check_launch(const char* op);            // cudaGetLastError -> status
int sm_count();                                    // SMs of the current device (cached)

// ---- formats ------------------------------------------------------------------------------
enum Format : int { F_Q4_0 = 0, F_Q8_0, F_Q6_K, F_MXFP8, F_NVFP4, F_MXFP4, F_COUNT };
int parse_format(const char* name);                // -1 if unknown
__host__ __device__ constexpr int block_k_of(int f) {
  return f == F_Q6_K ? 256 : (f == F_NVFP4 ? 16 : 32);
}
__host__ __device__ constexpr int block_bytes_of(int f) {
  return f == F_Q4_0 ? 18 : f == F_Q8_0 ? 34 : f == F_Q6_K ? 210 : f == F_MXFP8 ? 33
       : f == F_NVFP4 ? 9 : 17;
}

// ---- element types ------------------------------------------------------------------------
template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) {
  return __bfloat162float(v);
}
template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) {
  return __float2bfloat16_rn(v);
}

// ---- epilogue math (fp32; same formulas as the reference kernels) --------------------------
// erf by the 5-term Abramowitz-Stegun polynomial, then 0.5*v*(1+erf(v/sqrt2)).
__device__ __forceinline__ float gelu_erf_as(float v) {
  const float z = v * 0.70710678118654752440f;
  const float a = fabsf(z);
  const float t = 1.0f / (1.0f + 0.3275911f * a);
  const float poly =
      (((((1.061405429f * t + -1.453152027f) * t) + 1.421413741f) * t + -0.284496736f) * t +
       0.254829592f) * t;
  const float y = 1.0f - poly * expf(-a * a);
  return 0.5f * v * (1.0f + (z < 0.0f ? -y : y));
}
__device__ __forceinline__ float silu(float v) { return v / (1.0f + expf(-v)); }
__device__ __forceinline__ float apply_act(float v, int activation) {
  if (activation == 1) return gelu_erf_as(v);
  if (activation == 2) return silu(v);
  return v;
}

// ---- RNG: stateless integer hash keyed by (seed, row, global vocab id) ----------------------
__device__ __forceinline__ float rng_uniform(uint32_t seed, uint32_t a, uint32_t b) {
  uint32_t x = seed * 0x9E3779B9u + a * 0x85EBCA77u + b * 0xC2B2AE3Du;
  x ^= x >> 16; x *= 0x7FEB352Du;
  x ^= x >> 15; x *= 0x846CA68Bu;
  x ^= x >> 16;
  return (float)(x >> 8) * (1.0f / 16777216.0f);
}
__device__ __forceinline__ float rng_gumbel(uint32_t seed, uint32_t a, uint32_t b) {
  const float u = fmaxf(rng_uniform(seed, a, b), 1e-20f);
  return -logf(-logf(u));
}

#define QX_NEG_INF (-3.4028234663852886e38f)

// (value descending, id ascending) ordering used by every selection on this path
__device__ __forceinline__ bool better(float v, int id, float bv, int bid) {
  return v > bv || (v == bv && id < bid);
}
__device__ __forceinline__ void warp_argmax(float& v, int& id) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, off);
    const int oi = __shfl_xor_sync(0xffffffffu, id, off);
    if (better(ov, oi, v, id)) { v = ov; id = oi; }
  }
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}

// ---- output quantizer encoders (fp32 arithmetic on already-rounded I/O-dtype values) ---------
// e4m3: nearest with halves rounded AWAY from zero, |x| >= 448 and NaN -> 0x7E, |x| < 2^-10 ->
// signed zero.  int8: round half away, clamp to +-127.
// Without a branch: adding half a step to the bits of |x| rounds the mantissa to 3 bits and carries into the
// exponent; below 2^-6 the code is |x| * 512 rounded (the sum truncated, so that no second rounding can cross
// a half).  33 instructions with four branches became 11.
__device__ __forceinline__ uint32_t e4m3_encode(float x) {
  const uint32_t sign = (x < 0.0f) ? 0x80u : 0u;
  const float a = fabsf(x);
  const uint32_t normal = ((__float_as_uint(a) + 0x80000u) >> 20) - 120u * 8u;
  const uint32_t small = (uint32_t)__float2int_rz(__fadd_rz(a * 512.0f, 0.5f));
  return sign | min(a < 0.015625f ? small : normal, 0x7Eu);
}

// ---- codes of pairs of finite values ----
// Both conversions below round ties to even where e4m3_encode and int8_encode go away from zero: with the last
// mantissa bit set a tie is none any more, and no other value is moved past a rounding boundary.
// e4m3_encode(v.x) | e4m3_encode(v.y) << 8; the sum with 0 drops the sign of -0
__device__ __forceinline__ uint32_t e4m3_encode2(float2 v) {
  const float2 u = __fadd2_rn(v, make_float2(0.f, 0.f));
  const float a = __uint_as_float(__float_as_uint(u.x) | 1u), b = __uint_as_float(__float_as_uint(u.y) | 1u);
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(b), "f"(a));
  return r;
}
// int8_encode of both, |v| < 127.5, as the low bytes of the two words: 1.5 * 2^23 + v holds v's integer there
__device__ __forceinline__ uint2 int8_encode2(float2 v) {
  const float2 m = __fadd2_rn(make_float2(__uint_as_float(__float_as_uint(v.x) | 1u), __uint_as_float(__float_as_uint(v.y) | 1u)),
                          make_float2(12582912.f, 12582912.f));
  return make_uint2(__float_as_uint(m.x), __float_as_uint(m.y));
}

__device__ __forceinline__ int int8_encode(float x) {
  float r = roundf(x);                                    // half away from zero
  r = fminf(fmaxf(r, -127.0f), 127.0f);
  return (int)r;
}

// exact ceil(log2(q)) for a positive finite fp32 q
__device__ __forceinline__ int ceil_log2(float q) {
  const uint32_t bits = __float_as_uint(q);
  int e = (int)((bits >> 23) & 0xFFu) - 127;
  if (bits & 0x7FFFFFu) e += 1;
  return e;
}

// One MXFP8 block {e8m0 exponent; 32 e4m3 codes} from the 32 values held one per lane of a full
// warp: scale 2^ceil(log2(amax / 448)) (amax > 0), an all-zero block stores exponent 127.
__device__ __forceinline__ void mxfp8_block_store(float v, int lane, uint8_t* __restrict__ block) {
  // largest magnitude as bits (one warp reduction; NaN does not choose the scale); 448 = 1.75 * 2^8, so
  // ceil(log2(amax / 448)) is the exponent of amax - 8, plus one when its mantissa is above 1.75 (the sum below
  // carries then); an infinity takes the largest scale
  const uint32_t top = __reduce_max_sync(0xffffffffu, v == v ? __float_as_uint(v) & 0x7FFFFFFFu : 0u);
  int code = 127;
  if (top != 0u) {
    const uint32_t t = max(top, __float_as_uint(1e-10f));
    code = t == 0x7F800000u ? 254 : (int)((t + 0x1FFFFFu) >> 23) - 8;
  }
  const float inv = __uint_as_float(max((uint32_t)(254 - code) << 23, 0x00400000u));     // 2^(127 - code)
  block[1 + lane] = (uint8_t)e4m3_encode(v * inv);
  if (lane == 0) block[0] = (uint8_t)code;
}

}  // namespace qx
