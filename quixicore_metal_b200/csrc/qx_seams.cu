// The seams that hand quantised activations to the projections:
//   * residual add + RMSNorm with an optional quantising tail
//     (kernels/norms/add_norm/add_norm.metal:26-65 plain, :181-218 static fp8, :220-265 per-row
//     dynamic fp8, :268-312 per-row int8, :327-392 per-128-block fp8 / int8 with optional
//     power-of-two scales);
//   * gated activation (SwiGLU, or the clamped alpha-scaled variant) straight to per-token or
//     per-group fp8 / per-token int8 codes (kernels/quantization/act_quant/act_quant.metal:26-160,
//     activation math include/metal/common/glu_eval.metal:49-66).
// Everything is computed in fp32 from the I/O-dtype inputs; the sum x + residual is written back
// rounded to the I/O dtype while the norm continues on the unrounded fp32 sum; the quantisers see
// the unrounded fp32 values, as in the reference.  One CTA per row, the row kept in shared memory.
#include "qx_common.cuh"
#include "qx_kernels.h"
#include "qx_stream.cuh"
#include <type_traits>

namespace qx {

constexpr int SEAM_THREADS = 256;

__device__ __forceinline__ float seam_block_reduce(float v, bool is_max, float* red) {
  v = is_max ? warp_max(v) : warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = red[0];
#pragma unroll
  for (int i = 1; i < SEAM_THREADS / 32; ++i) r = is_max ? fmaxf(r, red[i]) : r + red[i];
  return r;
}

// scale for an absolute maximum: amax / qmax, or (pow2) the next power of two at or above it
__device__ __forceinline__ float seam_scale(float amax, float qmax, int pow2) {
  if (pow2 && amax > 0.f) {
    const int e = min(max(ceil_log2(fmaxf(amax, 1e-10f) / qmax), -126), 127);   // >= -42 by the clamp on amax
    return __uint_as_float((uint32_t)(e + 127) << 23);
  }
  return amax / qmax;
}

// Elements move in 16-byte vectors (8 two-byte or 4 four-byte elements per load / store; codes as
// 8- or 4-byte words) when VEC > 1: D % VEC == 0 and 16-byte aligned rows, checked by the launcher.
template <typename T, int VEC>
__device__ __forceinline__ void seam_load(const T* __restrict__ p, size_t i, float (&v)[VEC]) {
  if constexpr (VEC == 1) {
    v[0] = to_f32<T>(p[i]);
  } else {
    T tmp[VEC];
    *reinterpret_cast<uint4*>(tmp) = *reinterpret_cast<const uint4*>(p + i);
#pragma unroll
    for (int e = 0; e < VEC; ++e) v[e] = to_f32<T>(tmp[e]);
  }
}
template <typename T, int VEC>
__device__ __forceinline__ void seam_store(T* __restrict__ p, size_t i, const float (&v)[VEC]) {
  if constexpr (VEC == 1) {
    p[i] = from_f32<T>(v[0]);
  } else {
    T tmp[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) tmp[e] = from_f32<T>(v[e]);
    *reinterpret_cast<uint4*>(p + i) = *reinterpret_cast<const uint4*>(tmp);
  }
}
// Position of row element c in the shared-memory copy of the row.  With 8-element vectors a thread
// owns 8 consecutive elements; keeping them contiguous would put consecutive lanes 32 bytes apart
// (bank conflicts on every access), so the two halves of a vector live in two planes of D / 2
// floats, each holding one float4 per vector: consecutive lanes, consecutive float4s.
template <int VEC>
__device__ __forceinline__ int seam_sidx(int c, int D) {
  if constexpr (VEC == 8) return ((c >> 2) & 1) * (D >> 1) + ((c >> 3) << 2) + (c & 3);
  else return c;
}
// the VEC elements from c (a multiple of VEC) to / from the shared row
template <int VEC>
__device__ __forceinline__ void seam_row_put(float* __restrict__ row, int c, int D, const float (&v)[VEC]) {
  if constexpr (VEC == 1) row[c] = v[0];
  else {
#pragma unroll
    for (int q = 0; q < VEC / 4; ++q)
      *reinterpret_cast<float4*>(row + seam_sidx<VEC>(c + 4 * q, D)) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
  }
}
template <int VEC>
__device__ __forceinline__ void seam_row_get(const float* __restrict__ row, int c, int D, float (&v)[VEC]) {
  if constexpr (VEC == 1) v[0] = row[c];
  else {
#pragma unroll
    for (int q = 0; q < VEC / 4; ++q) {
      const float4 f = *reinterpret_cast<const float4*>(row + seam_sidx<VEC>(c + 4 * q, D));
      v[4 * q] = f.x; v[4 * q + 1] = f.y; v[4 * q + 2] = f.z; v[4 * q + 3] = f.w;
    }
  }
}

template <int VEC>
__device__ __forceinline__ void seam_store_codes(uint8_t* __restrict__ p, size_t i, const float (&v)[VEC], bool int8) {
  uint8_t c[VEC];
#pragma unroll
  for (int e = 0; e < VEC; ++e) c[e] = int8 ? (uint8_t)(int8_t)int8_encode(v[e]) : (uint8_t)e4m3_encode(v[e]);
  if constexpr (VEC == 8) *reinterpret_cast<uint2*>(p + i) = *reinterpret_cast<const uint2*>(c);
  else if constexpr (VEC == 4) *reinterpret_cast<uint32_t*>(p + i) = *reinterpret_cast<const uint32_t*>(c);
  else p[i] = c[0];
}
// absolute maximum and codes of the group of G elements from column c0, by one warp
template <int VEC>
__device__ __forceinline__ float seam_group_amax(const float* __restrict__ row, int c0, int G, int D, int lane) {
  float gm = 0.f;
  if constexpr (VEC > 1) {
    for (int i4 = lane; i4 < G / 4; i4 += 32) {
      const float4 f = *reinterpret_cast<const float4*>(row + seam_sidx<VEC>(c0 + 4 * i4, D));
      gm = fmaxf(fmaxf(gm, fmaxf(fabsf(f.x), fabsf(f.y))), fmaxf(fabsf(f.z), fabsf(f.w)));
    }
  } else {
    for (int i = lane; i < G; i += 32) gm = fmaxf(gm, fabsf(row[c0 + i]));
  }
  return warp_max(gm);
}
template <int VEC>
__device__ __forceinline__ void seam_group_codes(const float* __restrict__ row, int c0, uint8_t* __restrict__ dst, int G,
                                                 int D, float q_inv, bool int8, int lane) {
  if constexpr (VEC > 1) {
    for (int i4 = lane; i4 < G / 4; i4 += 32) {
      const float4 f = *reinterpret_cast<const float4*>(row + seam_sidx<VEC>(c0 + 4 * i4, D));
      const float v[4] = {f.x * q_inv, f.y * q_inv, f.z * q_inv, f.w * q_inv};
      seam_store_codes<4>(dst, (size_t)4 * i4, v, int8);
    }
  } else {
    for (int i = lane; i < G; i += 32) {
      const float v[1] = {row[c0 + i] * q_inv};
      seam_store_codes<1>(dst, (size_t)i, v, int8);
    }
  }
}

// qmode: 0 none (y in T), 1 fp8 static (inv_scale given), 2 fp8 per row, 3 int8 per row,
//        4 fp8 per group of G, 5 int8 per group of G.  scale: (rows,) or (rows, D/G).
template <typename T, int VEC>
__global__ void __launch_bounds__(SEAM_THREADS)
rms_norm_add_kernel(const T* __restrict__ x, const T* __restrict__ residual, const T* __restrict__ weight,
                    T* __restrict__ y, uint8_t* __restrict__ codes, T* __restrict__ res_out,
                    float* __restrict__ scale, int D, float eps, int qmode, float inv_static, int G, int pow2) {
  extern __shared__ __align__(16) float row[]; // D floats: x + residual, then the normalised row
  __shared__ float red[SEAM_THREADS / 32];
  const size_t base = (size_t)blockIdx.x * D;
  float ss = 0.f;
  for (int i = threadIdx.x * VEC; i < D; i += SEAM_THREADS * VEC) {
    float a[VEC], b[VEC], h[VEC];
    seam_load<T, VEC>(x, base + i, a);
    seam_load<T, VEC>(residual, base + i, b);
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      h[e] = a[e] + b[e];
      ss = fmaf(h[e], h[e], ss);
    }
    seam_row_put<VEC>(row, i, D, h);
    seam_store<T, VEC>(res_out, base + i, h);
  }
  const float ms = seam_block_reduce(ss, false, red) / (float)D;
  const float inv = rsqrtf(ms + eps);
  float amax = 0.f;
  for (int i = threadIdx.x * VEC; i < D; i += SEAM_THREADS * VEC) {
    float w[VEC], v[VEC];
    seam_load<T, VEC>(weight, (size_t)i, w);
    seam_row_get<VEC>(row, i, D, v);
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      v[e] = (v[e] * inv) * w[e];
      amax = fmaxf(amax, fabsf(v[e]));
    }
    seam_row_put<VEC>(row, i, D, v);
  }
  if (qmode == 0) {
    for (int i = threadIdx.x * VEC; i < D; i += SEAM_THREADS * VEC) {
      float v[VEC];
      seam_row_get<VEC>(row, i, D, v);
      seam_store<T, VEC>(y, base + i, v);
    }
    return;
  }
  if (qmode <= 3) {
    float q_inv = inv_static;
    if (qmode >= 2) {
      amax = seam_block_reduce(amax, true, red);
      const float s = amax / (qmode == 2 ? 448.0f : 127.0f);
      q_inv = s > 0.f ? 1.0f / s : 0.f;
      if (threadIdx.x == 0) scale[blockIdx.x] = s;
    }
    for (int i = threadIdx.x * VEC; i < D; i += SEAM_THREADS * VEC) {
      float v[VEC];
      seam_row_get<VEC>(row, i, D, v);
#pragma unroll
      for (int e = 0; e < VEC; ++e) v[e] *= q_inv;
      seam_store_codes<VEC>(codes, base + i, v, qmode == 3);
    }
    return;
  }
  // per group: a warp takes whole groups
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ngroups = D / G;
  const float qmax = qmode == 4 ? 448.0f : 127.0f;
  for (int g = warp; g < ngroups; g += SEAM_THREADS / 32) {
    const float gm = seam_group_amax<VEC>(row, g * G, G, D, lane);
    const float s = seam_scale(gm, qmax, qmode == 4 ? pow2 : 0);
    const float q_inv = s > 0.f ? 1.0f / s : 0.f;
    seam_group_codes<VEC>(row, g * G, codes + base + (size_t)g * G, G, D, q_inv, qmode == 5, lane);
    if (lane == 0) scale[(size_t)blockIdx.x * ngroups + g] = s;
  }
}

// act: 0 silu(x) * gate, 1 clamped: x <- min(x, limit), gate <- clamp(gate, +-limit),
// x * sigmoid(alpha x) * (1 + gate)
__device__ __forceinline__ float gated_act(int act, float x0, float x1, float alpha, float limit) {
  if (act == 1) {
    x0 = fminf(x0, limit);
    x1 = fmaxf(fminf(x1, limit), -limit);
    return (x0 / (1.0f + expf(-x0 * alpha))) * (1.0f + x1);
  }
  return (x0 / (1.0f + expf(-x0))) * x1;
}

// The same for P pairs.  exp(-t) = 2^(f - n), n the integer next to t log2(e) and f = n - t log2(e) by two fused
// multiply-adds (Cody and Waite: the first is exact but for its last bit, the second adds the constant's tail).  The
// quotient x / d, d = 1 + exp(-t), as one reciprocal estimate and one residual correction (Markstein: q = x r,
// q += (x - q d) r),
// right to half a unit of the last place but for values next to a rounding boundary.  d is in [1, 2^93) for |t| <= 64;
// a vector with a larger |t| (an infinity among them) takes expf and the plain divisions.
template <int P>
__device__ __forceinline__ void gated_act_pairs(int act, const float2 (&x)[P], const float2 (&g)[P], float alpha, float limit,
                                                float2 (&v)[P]) {
  float2 xs[P], gs[P], t[P];
  float big = 0.f;
#pragma unroll
  for (int p = 0; p < P; ++p) {
    xs[p] = t[p] = x[p];
    gs[p] = g[p];
    if (act == 1) {
      xs[p] = make_float2(fminf(x[p].x, limit), fminf(x[p].y, limit));
      gs[p] = make_float2(1.0f + fmaxf(fminf(g[p].x, limit), -limit), 1.0f + fmaxf(fminf(g[p].y, limit), -limit));
      t[p] = make_float2(xs[p].x * alpha, xs[p].y * alpha);
    }
    big = fmaxf(fmaxf(big, fabsf(t[p].x)), fabsf(t[p].y));
  }
  if (big > 64.f) {
#pragma unroll
    for (int p = 0; p < P; ++p)
      v[p] = make_float2((xs[p].x / (1.0f + expf(-t[p].x))) * gs[p].x, (xs[p].y / (1.0f + expf(-t[p].y))) * gs[p].y);
    return;
  }
  constexpr float L = 1.44269502162933349609375f, LT = 1.9259629911e-8f;   // log2(e) = L + LT
#pragma unroll
  for (int p = 0; p < P; ++p) {
    const float2 m = __ffma2_rn(t[p], make_float2(L, L), make_float2(12582912.f, 12582912.f));      // n in its low bits
    const float2 n = __fadd2_rn(m, make_float2(-12582912.f, -12582912.f));
    const float2 f = __ffma2_rn(t[p], make_float2(-LT, -LT), __ffma2_rn(t[p], make_float2(-L, -L), n));
    float2 e, rc;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(f.x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(f.y));
    e.x = __uint_as_float(__float_as_uint(e.x) - (__float_as_uint(m.x) << 23));
    e.y = __uint_as_float(__float_as_uint(e.y) - (__float_as_uint(m.y) << 23));
    const float2 d = __fadd2_rn(e, make_float2(1.f, 1.f));
    const float2 nd = __ffma2_rn(e, make_float2(-1.f, -1.f), make_float2(-1.f, -1.f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rc.x) : "f"(d.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rc.y) : "f"(d.y));
    const float2 q = __fmul2_rn(xs[p], rc);
    v[p] = __fmul2_rn(__ffma2_rn(__ffma2_rn(q, nd, xs[p]), rc, q), gs[p]);
  }
}

// qmode: 2 fp8 per row, 3 int8 per row, 4 fp8 per group of G (pow2: power-of-two scales)
template <typename T, int VEC>
__global__ void __launch_bounds__(SEAM_THREADS)
silu_mul_quant_kernel(const T* __restrict__ x, const T* __restrict__ gate, uint8_t* __restrict__ codes,
                      float* __restrict__ scale, int D, int act, float alpha, float limit, int qmode, int G,
                      int pow2) {
  extern __shared__ __align__(16) float row[];
  __shared__ float red[SEAM_THREADS / 32];
  const size_t base = (size_t)blockIdx.x * D;
  float amax = 0.f;
  for (int i = threadIdx.x * VEC; i < D; i += SEAM_THREADS * VEC) {
    float a[VEC], b[VEC];
    seam_load<T, VEC>(x, base + i, a);
    seam_load<T, VEC>(gate, base + i, b);
    float v[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      v[e] = gated_act(act, a[e], b[e], alpha, limit);
      amax = fmaxf(amax, fabsf(v[e]));
    }
    seam_row_put<VEC>(row, i, D, v);
  }
  if (qmode <= 3) {
    amax = seam_block_reduce(amax, true, red);
    const float s = amax / (qmode == 2 ? 448.0f : 127.0f);
    const float q_inv = s > 0.f ? 1.0f / s : 0.f;
    if (threadIdx.x == 0) scale[blockIdx.x] = s;
    for (int i = threadIdx.x * VEC; i < D; i += SEAM_THREADS * VEC) {
      float v[VEC];
      seam_row_get<VEC>(row, i, D, v);
#pragma unroll
      for (int e = 0; e < VEC; ++e) v[e] *= q_inv;
      seam_store_codes<VEC>(codes, base + i, v, qmode == 3);
    }
    return;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ngroups = D / G;
  for (int g = warp; g < ngroups; g += SEAM_THREADS / 32) {
    const float gm = seam_group_amax<VEC>(row, g * G, G, D, lane);
    const float s = seam_scale(gm, 448.0f, pow2);
    const float q_inv = s > 0.f ? 1.0f / s : 0.f;
    seam_group_codes<VEC>(row, g * G, codes + base + (size_t)g * G, G, D, q_inv, false, lane);
    if (lane == 0) scale[(size_t)blockIdx.x * ngroups + g] = s;
  }
}

// ---- rows held in registers -------------------------------------------------------------------------
// R vectors of 16 bytes per thread and operand, vector r of thread i at element (r * threads + i) * VEC.  What bounds
// these is instructions first (32 and 43 per element before pairs and hardware code conversions) and memory next: with
// one CTA per row the loads, the reductions and the stores of a row follow one another and
// too few rows overlap.  RING: persistent CTAs, each with a ring of SEAM_STAGES rows filled by bulk copies ahead of the
// arithmetic; without it (no more rows than resident CTAs) a CTA loads its one row directly.  4096 rows of 8192 bf16 to
// fp8 per row on B200, shared-memory rows -> these: rms_norm_add 49.5 -> 41 us (5.7 TB/s), silu_mul 54.8 -> 44 us.
constexpr int SEAM_REG_THREADS = 512;
constexpr int SEAM_STAGES = 3;

// `red`: one array per reduction of a row; a barrier between the rows keeps them apart
__device__ __forceinline__ float seam_reg_reduce(float v, bool is_max, float* red) {
  v = is_max ? warp_max(v) : warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  v = lane < (int)(blockDim.x >> 5) ? red[lane] : 0.f;
  return is_max ? warp_max(v) : warp_sum(v);
}

template <typename T, int VEC, int R>
__device__ __forceinline__ void seam_reg_load(const T* __restrict__ p, int D, uint4 (&raw)[R]) {
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = (r * (int)blockDim.x + (int)threadIdx.x) * VEC;
    raw[r] = i < D ? __ldg(reinterpret_cast<const uint4*>(p + i)) : make_uint4(0u, 0u, 0u, 0u);
  }
}
// body(row, a, b) for every row of this CTA, a and b this thread's vectors of the row of either operand
template <typename T, int R, bool RING, class Body>
__device__ __forceinline__ void seam_rows(const T* __restrict__ pa, const T* __restrict__ pb, int rows, int D, int* err,
                                          Body&& body) {
  constexpr int VEC = 16 / (int)sizeof(T);
  uint4 a[R], b[R];
  if constexpr (!RING) {
    seam_reg_load<T, VEC, R>(pa + (size_t)blockIdx.x * D, D, a);
    seam_reg_load<T, VEC, R>(pb + (size_t)blockIdx.x * D, D, b);
    body((int)blockIdx.x, a, b);
  } else {
    extern __shared__ __align__(128) uint8_t seam_ring[];           // [stage][operand][D]
    __shared__ __align__(8) uint64_t bars[SEAM_STAGES];
    const uint32_t bytes = (uint32_t)D * (uint32_t)sizeof(T);
    auto issue = [&](int row, int stage) {
      const uint32_t bar = smem_u32(bars + stage), dst = smem_u32(seam_ring) + (uint32_t)stage * 2u * bytes;
      mbar_arrive_expect_tx(bar, 2u * bytes);
      bulk_g2s(dst, pa + (size_t)row * D, bytes, bar);
      bulk_g2s(dst + bytes, pb + (size_t)row * D, bytes, bar);
    };
    if (threadIdx.x == 0) {
      for (int i = 0; i < SEAM_STAGES; ++i) mbar_init(smem_u32(bars + i), 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      for (int i = 0; i < SEAM_STAGES; ++i)
        if ((long long)blockIdx.x + (long long)i * gridDim.x < rows) issue((int)(blockIdx.x + i * gridDim.x), i);
    }
    __syncthreads();
    int stage = 0;
    uint32_t parity = 0;
    bool dead = false;                                               // a wait ran out: no further wait, no further copy
    for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
      if (!dead) dead = !mbar_wait(smem_u32(bars + stage), parity, err);
      const uint4* sa = reinterpret_cast<const uint4*>(seam_ring + (size_t)stage * 2 * bytes);
      const uint4* sb = reinterpret_cast<const uint4*>(seam_ring + (size_t)(stage * 2 + 1) * bytes);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int i = r * (int)blockDim.x + (int)threadIdx.x;
        a[r] = i * VEC < D ? sa[i] : make_uint4(0u, 0u, 0u, 0u);
        b[r] = i * VEC < D ? sb[i] : make_uint4(0u, 0u, 0u, 0u);
      }
      __syncthreads();                                               // the stage is read, and the reductions of the row before are
      const long long next = row + (long long)SEAM_STAGES * gridDim.x;
      if (threadIdx.x == 0 && next < rows && !dead) issue((int)next, stage);
      if (++stage == SEAM_STAGES) { stage = 0; parity ^= 1u; }
      body((int)row, a, b);
    }
  }
}
template <typename T, int P>
__device__ __forceinline__ void seam_widen(const uint4& raw, float2 (&v)[P]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int p = 0; p < P; ++p) {
    if constexpr (sizeof(T) == 4) v[p] = make_float2(__uint_as_float(w[2 * p]), __uint_as_float(w[2 * p + 1]));
    else if constexpr (std::is_same<T, __half>::value) v[p] = __half22float2(*reinterpret_cast<const __half2*>(&w[p]));
    else v[p] = make_float2(__uint_as_float(w[p] << 16), __uint_as_float(w[p] & 0xFFFF0000u));
  }
}
template <typename T, int P>
__device__ __forceinline__ void seam_store_pairs(T* __restrict__ dst, const float2 (&v)[P]) {
  uint32_t w[4];
#pragma unroll
  for (int p = 0; p < P; ++p) {
    if constexpr (sizeof(T) == 4) { w[2 * p] = __float_as_uint(v[p].x); w[2 * p + 1] = __float_as_uint(v[p].y); }
    else if constexpr (std::is_same<T, __half>::value) { const __half2 h = __floats2half2_rn(v[p].x, v[p].y); w[p] = *reinterpret_cast<const uint32_t*>(&h); }
    else { const __nv_bfloat162 h = __floats2bfloat162_rn(v[p].x, v[p].y); w[p] = *reinterpret_cast<const uint32_t*>(&h); }
  }
  *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
}
// codes of v * q_inv
template <int P>
__device__ __forceinline__ void seam_store_codes_pairs(uint8_t* __restrict__ dst, const float2 (&v)[P], float q_inv, bool int8) {
  float2 u[P], z = make_float2(0.f, 0.f);
#pragma unroll
  for (int p = 0; p < P; ++p) {
    u[p] = __fmul2_rn(v[p], make_float2(q_inv, q_inv));
    z = __ffma2_rn(u[p], make_float2(0.f, 0.f), z);                      // NaN once a value is not finite
  }
  if (!(z.x + z.y == 0.f)) {
    float s[2 * P];
#pragma unroll
    for (int p = 0; p < P; ++p) { s[2 * p] = u[p].x; s[2 * p + 1] = u[p].y; }
    seam_store_codes<2 * P>(dst, 0, s, int8);
    return;
  }
  uint32_t c[P / 2];
#pragma unroll
  for (int q = 0; q < P / 2; ++q) {
    if (int8) {
      const uint2 a = int8_encode2(u[2 * q]), b = int8_encode2(u[2 * q + 1]);
      c[q] = __byte_perm(__byte_perm(a.x, a.y, 0x0040), __byte_perm(b.x, b.y, 0x0040), 0x5410);
    } else {
      c[q] = e4m3_encode2(u[2 * q]) | e4m3_encode2(u[2 * q + 1]) << 16;
    }
  }
  if constexpr (P == 4) *reinterpret_cast<uint2*>(dst) = make_uint2(c[0], c[1]);
  else *reinterpret_cast<uint32_t*>(dst) = c[0];
}

// qmode 1 .. 5 of the values in registers; a group is G / VEC lanes of a warp (a power of two)
template <int VEC, int R>
__device__ __forceinline__ void seam_reg_quant(int row, const float2 (&v)[R][VEC / 2], uint8_t* __restrict__ codes,
                                               float* __restrict__ scale, int D, int qmode, float inv_static, int G, int pow2,
                                               float* red) {
  float am[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    am[r] = 0.f;
    if (qmode == 1) continue;
#pragma unroll
    for (int p = 0; p < VEC / 2; ++p) am[r] = fmaxf(fmaxf(am[r], fabsf(v[r][p].x)), fabsf(v[r][p].y));
  }
  float q_inv = inv_static;
  if (qmode == 2 || qmode == 3) {
#pragma unroll
    for (int r = 1; r < R; ++r) am[0] = fmaxf(am[0], am[r]);
    const float s = seam_reg_reduce(am[0], true, red) / (qmode == 2 ? 448.0f : 127.0f);
    q_inv = s > 0.f ? 1.0f / s : 0.f;
    if (threadIdx.x == 0) scale[row] = s;
  }
  const float qmax = qmode == 5 ? 127.0f : 448.0f;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = (r * (int)blockDim.x + (int)threadIdx.x) * VEC;
    if (qmode >= 4) {
      for (int o = 1; o < G / VEC; o <<= 1) am[r] = fmaxf(am[r], __shfl_xor_sync(0xffffffffu, am[r], o));
      const float s = seam_scale(am[r], qmax, qmode == 4 ? pow2 : 0);
      q_inv = s > 0.f ? 1.0f / s : 0.f;
      if (i < D && i % G == 0) scale[(size_t)row * (D / G) + i / G] = s;
    }
    if (i < D) seam_store_codes_pairs<VEC / 2>(codes + (size_t)row * D + i, v[r], q_inv, qmode == 3 || qmode == 5);
  }
}

template <typename T, int R, bool RING>
__global__ void __launch_bounds__(SEAM_REG_THREADS, R <= 2 ? 2 : 1)
rms_norm_add_reg_kernel(const T* __restrict__ x, const T* __restrict__ residual, const T* __restrict__ weight,
                        T* __restrict__ y, uint8_t* __restrict__ codes, T* __restrict__ res_out, float* __restrict__ scale,
                        int rows, int D, float eps, int qmode, float inv_static, int G, int pow2, int* err) {
  constexpr int VEC = 16 / (int)sizeof(T);
  __shared__ float red[2][SEAM_REG_THREADS / 32];
  uint4 wv[R];
  seam_reg_load<T, VEC, R>(weight, D, wv);
  seam_rows<T, R, RING>(x, residual, rows, D, err, [&](int row, const uint4 (&xa)[R], const uint4 (&xb)[R]) {
    const size_t base = (size_t)row * D;
    float2 v[R][VEC / 2], ss = make_float2(0.f, 0.f);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = (r * (int)blockDim.x + (int)threadIdx.x) * VEC;
      float2 a[VEC / 2], b[VEC / 2];
      seam_widen<T>(xa[r], a);
      seam_widen<T>(xb[r], b);
#pragma unroll
      for (int p = 0; p < VEC / 2; ++p) {
        v[r][p] = __fadd2_rn(a[p], b[p]);
        ss = __ffma2_rn(v[r][p], v[r][p], ss);
      }
      if (i < D) seam_store_pairs<T>(res_out + base + i, v[r]);
    }
    const float inv = rsqrtf(seam_reg_reduce(ss.x + ss.y, false, red[0]) / (float)D + eps);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = (r * (int)blockDim.x + (int)threadIdx.x) * VEC;
      float2 w[VEC / 2];
      seam_widen<T>(wv[r], w);
#pragma unroll
      for (int p = 0; p < VEC / 2; ++p) v[r][p] = __fmul2_rn(__fmul2_rn(v[r][p], make_float2(inv, inv)), w[p]);
      if (qmode == 0 && i < D) seam_store_pairs<T>(y + base + i, v[r]);
    }
    if (qmode != 0) seam_reg_quant<VEC, R>(row, v, codes, scale, D, qmode, inv_static, G, pow2, red[1]);
  });
}

template <typename T, int R, bool RING>
__global__ void __launch_bounds__(SEAM_REG_THREADS, R <= 2 ? 2 : 1)
silu_mul_quant_reg_kernel(const T* __restrict__ x, const T* __restrict__ gate, uint8_t* __restrict__ codes,
                          float* __restrict__ scale, int rows, int D, int act, float alpha, float limit, int qmode, int G,
                          int pow2, int* err) {
  constexpr int VEC = 16 / (int)sizeof(T);
  __shared__ float red[SEAM_REG_THREADS / 32];
  seam_rows<T, R, RING>(x, gate, rows, D, err, [&](int row, const uint4 (&xa)[R], const uint4 (&xb)[R]) {
    float2 v[R][VEC / 2];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float2 a[VEC / 2], b[VEC / 2];
      seam_widen<T>(xa[r], a);
      seam_widen<T>(xb[r], b);
      gated_act_pairs<VEC / 2>(act, a, b, alpha, limit, v[r]);
    }
    seam_reg_quant<VEC, R>(row, v, codes, scale, D, qmode, 0.f, G, pow2, red);
  });
}

// Vectors per thread for a row of D elements, 0 where the row has to lie in shared memory: rows past 4 vectors for each
// of 512 threads, unaligned ones, and groups that are not a power of two of lanes.  2 as long as that is enough: more
// threads per SM stay resident than with 4.
static int seam_reg_vectors(int64_t D, int vec, int qmode, int G) {
  if (D % vec != 0 || D > 4LL * vec * SEAM_REG_THREADS) return 0;
  const int lanes = qmode >= 4 ? (G % vec == 0 ? G / vec : 0) : 1;
  if (lanes < 1 || lanes > 32 || (lanes & (lanes - 1)) != 0) return 0;
  return D <= 2LL * vec * SEAM_REG_THREADS ? 2 : 4;
}
// Threads, CTAs and shared memory of such a launch.  Resident CTAs: 1024 threads (64 registers each, R = 2), and rings
// that fit the SM.  A grid no larger than that has one row per CTA and needs no ring.
struct SeamLaunch { int R; bool ring; unsigned threads, grid; size_t smem; };
static SeamLaunch seam_launch(int64_t rows, int64_t D, int es, int R) {
  SeamLaunch l{R, false, 0, (unsigned)rows, 0};
  const int64_t vecs = D / (16 / es);
  l.threads = (unsigned)((vecs + 32 * R - 1) / (32 * R)) * 32u;
  const size_t ring = (size_t)SEAM_STAGES * 2 * D * es;
  int64_t per_sm = (R == 2 ? 1024 : 512) / l.threads, fit = (int64_t)((size_t)220 * 1024 / (ring + 1536));
  if (per_sm > fit) per_sm = fit;
  if (per_sm >= 1 && rows > per_sm * sm_count() && device_error_flag() != nullptr) {
    l.ring = true;
    l.grid = (unsigned)(per_sm * sm_count());
    l.smem = ring;
  }
  return l;
}

template <typename K>
static bool seam_smem(K kernel, size_t bytes) {
  if (bytes <= 48 * 1024) return true;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess;
}

bool launch_rms_norm_add(cudaStream_t st, qx_dtype dtype, const void* x, const void* residual, const void* weight,
                         void* y, void* codes, void* res_out, float* scale, int64_t rows, int64_t D, float eps,
                         int qmode, float inv_static, int G, int pow2) {
  const size_t smem = (size_t)D * 4;
  if (smem > 200 * 1024) return false;
#define QX_NORM(T) \
  { constexpr int V = 16 / (int)sizeof(T); \
    const bool vec = D % V == 0 && (G <= 0 || G % 4 == 0) && \
        ((((uintptr_t)x | (uintptr_t)residual | (uintptr_t)weight | (uintptr_t)y | (uintptr_t)res_out | (uintptr_t)codes) & 15) == 0); \
    const int R = vec ? seam_reg_vectors(D, V, qmode, G) : 0; \
    const SeamLaunch l = R ? seam_launch(rows, D, (int)sizeof(T), R) : SeamLaunch{}; \
    auto reg = [&](auto kernel) { \
      if (!seam_smem(kernel, l.smem)) { cudaGetLastError(); return false; } \
      kernel<<<l.grid, l.threads, l.smem, st>>>((const T*)x, (const T*)residual, (const T*)weight, (T*)y, (uint8_t*)codes, \
          (T*)res_out, scale, (int)rows, (int)D, eps, qmode, inv_static, G, pow2, device_error_flag()); \
      return true; \
    }; \
    if (R) { \
      if (!(R == 2 ? (l.ring ? reg(rms_norm_add_reg_kernel<T, 2, true>) : reg(rms_norm_add_reg_kernel<T, 2, false>)) \
                   : (l.ring ? reg(rms_norm_add_reg_kernel<T, 4, true>) : reg(rms_norm_add_reg_kernel<T, 4, false>)))) return false; \
    } else if (vec) { \
      if (!seam_smem(rms_norm_add_kernel<T, V>, smem)) { cudaGetLastError(); return false; } \
      rms_norm_add_kernel<T, V><<<(unsigned)rows, SEAM_THREADS, smem, st>>>((const T*)x, (const T*)residual, (const T*)weight, \
          (T*)y, (uint8_t*)codes, (T*)res_out, scale, (int)D, eps, qmode, inv_static, G, pow2); \
    } else { \
      if (!seam_smem(rms_norm_add_kernel<T, 1>, smem)) { cudaGetLastError(); return false; } \
      rms_norm_add_kernel<T, 1><<<(unsigned)rows, SEAM_THREADS, smem, st>>>((const T*)x, (const T*)residual, (const T*)weight, \
          (T*)y, (uint8_t*)codes, (T*)res_out, scale, (int)D, eps, qmode, inv_static, G, pow2); \
    } }
  if (dtype == QX_DTYPE_F32) QX_NORM(float)
  else if (dtype == QX_DTYPE_F16) QX_NORM(__half)
  else QX_NORM(__nv_bfloat16)
#undef QX_NORM
  note_launch();
  return true;
}

bool launch_silu_mul_quant(cudaStream_t st, qx_dtype dtype, const void* x, const void* gate, void* codes, float* scale,
                           int64_t rows, int64_t D, int act, float alpha, float limit, int qmode, int G, int pow2) {
  const size_t smem = (size_t)D * 4;
  if (smem > 200 * 1024) return false;
#define QX_ACT(T) \
  { constexpr int V = 16 / (int)sizeof(T); \
    const bool vec = D % V == 0 && (G <= 0 || G % 4 == 0) && ((((uintptr_t)x | (uintptr_t)gate | (uintptr_t)codes) & 15) == 0); \
    const int R = vec ? seam_reg_vectors(D, V, qmode, G) : 0; \
    const SeamLaunch l = R ? seam_launch(rows, D, (int)sizeof(T), R) : SeamLaunch{}; \
    auto reg = [&](auto kernel) { \
      if (!seam_smem(kernel, l.smem)) { cudaGetLastError(); return false; } \
      kernel<<<l.grid, l.threads, l.smem, st>>>((const T*)x, (const T*)gate, (uint8_t*)codes, scale, (int)rows, (int)D, act, \
          alpha, limit, qmode, G, pow2, device_error_flag()); \
      return true; \
    }; \
    if (R) { \
      if (!(R == 2 ? (l.ring ? reg(silu_mul_quant_reg_kernel<T, 2, true>) : reg(silu_mul_quant_reg_kernel<T, 2, false>)) \
                   : (l.ring ? reg(silu_mul_quant_reg_kernel<T, 4, true>) : reg(silu_mul_quant_reg_kernel<T, 4, false>)))) return false; \
    } else if (vec) { \
      if (!seam_smem(silu_mul_quant_kernel<T, V>, smem)) { cudaGetLastError(); return false; } \
      silu_mul_quant_kernel<T, V><<<(unsigned)rows, SEAM_THREADS, smem, st>>>((const T*)x, (const T*)gate, (uint8_t*)codes, scale, \
          (int)D, act, alpha, limit, qmode, G, pow2); \
    } else { \
      if (!seam_smem(silu_mul_quant_kernel<T, 1>, smem)) { cudaGetLastError(); return false; } \
      silu_mul_quant_kernel<T, 1><<<(unsigned)rows, SEAM_THREADS, smem, st>>>((const T*)x, (const T*)gate, (uint8_t*)codes, scale, \
          (int)D, act, alpha, limit, qmode, G, pow2); \
    } }
  if (dtype == QX_DTYPE_F32) QX_ACT(float)
  else if (dtype == QX_DTYPE_F16) QX_ACT(__half)
  else QX_ACT(__nv_bfloat16)
#undef QX_ACT
  note_launch();
  return true;
}

}  // namespace qx
