// Shape-generic decode projections in fp32 arithmetic: the path of fp32 activations and of every 16-bit call
// whose shape or alignment the tensor-core kernels do not take.  Correct for any K % block_k == 0.
//
// What bounds it: latency (a 4096 x 1536 q4_0 matrix is 3.5 MB, 0.5 us of HBM time) and, for larger ones, the
// issue slots of decode + FMA.  So everything a lane needs for a step is asked for at once and coalesced:
// four lanes share a 32-column unit - a lane holds 8 weights of it, two groups of four consecutive columns, so
// that the activations are two vector loads - a warp covers 256 columns of R rows per step, and the warps of a
// CTA share the steps of a row when there are too few rows to fill the GPU.  The scale goes into the weights
// (exact products, four packed multiplications per 8 weights): a code times a large activation, or a large scale times
// the sum of eight products, can leave fp32 where the weight times the activation does not.  One warp per row with a 32-column span per lane (scalar, strided activation loads): 30.7 us for
// that matrix at one row with the full epilogue, now 4.5 to 5.
#include "qx_formats.cuh"
#include "qx_kernels.h"
#include "qx_stream.cuh"

namespace qx {

namespace {

// 4 / 8 bytes at any address, from the aligned words that hold them (no word without a wanted byte is read)
__device__ __forceinline__ uint32_t ldg4(const uint8_t* p) {
  const uint32_t* b = reinterpret_cast<const uint32_t*>((uintptr_t)p & ~(uintptr_t)3);
  const uint32_t sh = (uint32_t)((uintptr_t)p & 3) * 8u;
  const uint32_t lo = __ldg(b), hi = sh ? __ldg(b + 1) : 0u;
  return __funnelshift_r(lo, hi, sh);
}
__device__ __forceinline__ uint2 ldg8(const uint8_t* p) {
  const uint32_t* b = reinterpret_cast<const uint32_t*>((uintptr_t)p & ~(uintptr_t)3);
  const uint32_t sh = (uint32_t)((uintptr_t)p & 3) * 8u;
  const uint32_t w0 = __ldg(b), w1 = __ldg(b + 1), w2 = sh ? __ldg(b + 2) : 0u;
  return make_uint2(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh));
}
__device__ __forceinline__ float ldg_f16(const uint8_t* p) {          // 2-byte aligned
  return __half2float(__ushort_as_half(__ldg(reinterpret_cast<const uint16_t*>(p))));
}
__device__ __forceinline__ uint32_t e4m3_pair_bits(uint32_t v) {      // codes at [15:8], [31:24] -> f16 pair of value * 2^-8
  return ((v >> 1) & 0x3F803F80u) | (v & 0x80008000u);
}

// The 8 weights of lane quarter t of 32-column unit u: raw() loads, weights() gives them, scaled.
// cols(): first columns (inside the unit) of weights 0..3 and 4..7.
template <int FMT> struct Lane8 {
  uint32_t a, b, c, d;                             // code words (q6_K: low nibbles a, b and high bits c, d)
  float scale;
  __device__ __forceinline__ static int first(int t) {
    return FMT == F_Q4_0 || FMT == F_MXFP4 ? 4 * t : (FMT == F_NVFP4 ? 16 * (t >> 1) + 4 * (t & 1) : 8 * t);
  }
  static constexpr int GAP = FMT == F_Q4_0 || FMT == F_MXFP4 ? 16 : (FMT == F_NVFP4 ? 8 : 4);

  __device__ __forceinline__ void raw(const uint8_t* __restrict__ row, int u, int t) {
    if constexpr (FMT == F_Q4_0) {
      const uint8_t* p = row + (size_t)u * 18;
      a = ldg4(p + 2 + 4 * t); scale = ldg_f16(p);
    } else if constexpr (FMT == F_MXFP4) {
      const uint8_t* p = row + (size_t)u * 17;
      a = ldg4(p + 1 + 4 * t); scale = e8m0_to_f32(__ldg(p));
    } else if constexpr (FMT == F_NVFP4) {
      const uint8_t* p = row + (size_t)(2 * u + (t >> 1)) * 9;
      a = ldg4(p + 1 + 4 * (t & 1)); scale = e4m3_to_f32(__ldg(p));
    } else if constexpr (FMT == F_Q8_0) {
      const uint8_t* p = row + (size_t)u * 34;
      const uint2 v = ldg8(p + 2 + 8 * t);
      a = v.x; b = v.y; scale = ldg_f16(p);
    } else if constexpr (FMT == F_MXFP8) {
      const uint8_t* p = row + (size_t)u * 33;
      const uint2 v = ldg8(p + 1 + 8 * t);
      a = v.x; b = v.y; scale = e8m0_to_f32(__ldg(p));
    } else {
      const uint8_t* p = row + (size_t)(u >> 3) * 210;
      const int ch = (u >> 2) & 1, g = u & 3;      // 128-column half, 32-column quarter of it
      const uint2 q = ldg8(p + 64 * ch + 32 * (g & 1) + 8 * t), h = ldg8(p + 128 + 32 * ch + 8 * t);
      const int qs = 4 * (g >> 1), hs = 2 * g;
      a = q.x >> qs; b = q.y >> qs; c = h.x >> hs; d = h.y >> hs;
      scale = ldg_f16(p + 208) * (float)(int)(int8_t)__ldg(p + 192 + 8 * ch + 2 * g + (t >> 1));
    }
  }
  __device__ __forceinline__ static void pair(uint32_t h, float& x, float& y) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
    x = f.x; y = f.y;
  }
  // bytes of c4 (each a small integer) minus `off`, in order
  __device__ __forceinline__ static void ints(uint32_t c4, uint32_t off2, float* w) {
    pair(h2sub(__byte_perm(c4, 0x64646464u, 0x4140), off2), w[0], w[1]);
    pair(h2sub(__byte_perm(c4, 0x64646464u, 0x4342), off2), w[2], w[3]);
  }
  __device__ __forceinline__ void weights(float (&w)[8]) const {
    if constexpr (FMT == F_Q4_0) {
      ints(a & 0x0F0F0F0Fu, 0x64086408u, w);
      ints((a >> 4) & 0x0F0F0F0Fu, 0x64086408u, w + 4);
    } else if constexpr (FMT == F_MXFP4 || FMT == F_NVFP4) {
      pair(cvt_e2m1x2<0>(a), w[0], w[4]); pair(cvt_e2m1x2<1>(a), w[1], w[5]);
      pair(cvt_e2m1x2<2>(a), w[2], w[6]); pair(cvt_e2m1x2<3>(a), w[3], w[7]);
    } else if constexpr (FMT == F_Q8_0) {
      ints(a ^ 0x80808080u, 0x64806480u, w);
      ints(b ^ 0x80808080u, 0x64806480u, w + 4);
    } else if constexpr (FMT == F_MXFP8) {
      // * 256 in f16 (at most 480): a scale of 2^120 and more times 256 is none in fp32
      pair(h2mul(e4m3_pair_bits(__byte_perm(a, 0u, 0x1404)), 0x5C005C00u), w[0], w[1]);
      pair(h2mul(e4m3_pair_bits(__byte_perm(a, 0u, 0x3424)), 0x5C005C00u), w[2], w[3]);
      pair(h2mul(e4m3_pair_bits(__byte_perm(b, 0u, 0x1404)), 0x5C005C00u), w[4], w[5]);
      pair(h2mul(e4m3_pair_bits(__byte_perm(b, 0u, 0x3424)), 0x5C005C00u), w[6], w[7]);
    } else {
      ints((a & 0x0F0F0F0Fu) | ((c << 4) & 0x30303030u), 0x64206420u, w);
      ints((b & 0x0F0F0F0Fu) | ((d << 4) & 0x30303030u), 0x64206420u, w + 4);
    }
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const float2 v = __fmul2_rn(make_float2(w[i], w[i + 1]), make_float2(scale, scale));
      w[i] = v.x; w[i + 1] = v.y;
    }
  }
};

// four consecutive activations; vec: the address is aligned for one vector load
template <typename T>
__device__ __forceinline__ void load_x4(const T* __restrict__ p, bool vec, float* o) {
  if (vec) {
    if constexpr (sizeof(T) == 4) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(p));
      o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
    } else {
      const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
      const T* e = reinterpret_cast<const T*>(&v);
#pragma unroll
      for (int i = 0; i < 4; ++i) o[i] = to_f32<T>(e[i]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i] = to_f32<T>(p[i]);
  }
}

constexpr int GEN_WARPS = 8;

}  // namespace

// MB activation rows per pass (blockIdx.y); a warp owns R output rows (of both matrices when DUAL) and takes every
// S-th step of 256 columns, S = 1 << slog warps sharing the rows.
template <int FMT, typename T, int MB, int R, bool DUAL>
__global__ void __launch_bounds__(GEN_WARPS * 32)
gemv_generic_kernel(const T* __restrict__ x, const uint8_t* __restrict__ w0, const uint8_t* __restrict__ w1,
                    const T* __restrict__ bias0, const T* __restrict__ bias1, const T* __restrict__ residual,
                    T* __restrict__ y, int M, int K, int N, int activation, int use_bias, int use_residual, int slog,
                    int vec) {
  constexpr int BK = block_k_of(FMT), BB = block_bytes_of(FMT), NR = R * (DUAL ? 2 : 1);
  __shared__ float red[GEN_WARPS][NR * MB];
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = lane & 3;
  const int S = 1 << slog, slice = warp & (S - 1), grp = warp >> slog;
  const int n0 = (blockIdx.x * (GEN_WARPS >> slog) + grp) * R;
  const int m0 = blockIdx.y * MB, mcount = min(MB, M - m0);
  const size_t row_bytes = (size_t)(K / BK) * BB;
  const uint8_t* rows[NR];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const size_t at = (size_t)min(n0 + r, N - 1) * row_bytes;
    rows[r] = w0 + at;
    if constexpr (DUAL) rows[R + r] = w1 + at;
  }
  float acc[NR][MB];
#pragma unroll
  for (int r = 0; r < NR; ++r)
#pragma unroll
    for (int m = 0; m < MB; ++m) acc[r][m] = 0.f;

  const int first = Lane8<FMT>::first(t);
  constexpr int GAP = Lane8<FMT>::GAP;
#pragma unroll 2
  for (int k0 = slice * 256; k0 < K; k0 += S * 256) {
    const int u = (k0 >> 5) + (lane >> 2), col = 32 * u + first;
    if (col >= K) continue;                        // the lanes past the end of the last step
    Lane8<FMT> q[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) q[r].raw(rows[r], u, t);
    float xv[MB][8];
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      const T* xp = x + (size_t)(m0 + min(m, mcount - 1)) * K + col;
      load_x4<T>(xp, vec, xv[m]);
      load_x4<T>(xp + GAP, vec, xv[m] + 4);
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      float w[8];
      q[r].weights(w);
#pragma unroll
      for (int m = 0; m < MB; ++m) {
        float s = w[0] * xv[m][0];
#pragma unroll
        for (int i = 1; i < 8; ++i) s = fmaf(w[i], xv[m][i], s);
        acc[r][m] += s;
      }
    }
  }
#pragma unroll
  for (int r = 0; r < NR; ++r)
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      const float s = warp_sum(acc[r][m]);
      if (lane == 0) red[warp][r * MB + m] = s;
    }
  __syncthreads();
  // outputs of the CTA's row groups
  for (int i = threadIdx.x; i < (GEN_WARPS >> slog) * R * MB; i += GEN_WARPS * 32) {
    const int g = i / (R * MB), r = (i / MB) % R, m = i % MB;
    const int n = (blockIdx.x * (GEN_WARPS >> slog) + g) * R + r;
    if (n >= N || m >= mcount) continue;
    float v = 0.f, up = 0.f;
    for (int k = 0; k < S; ++k) {
      v += red[(g << slog) + k][r * MB + m];
      if constexpr (DUAL) up += red[(g << slog) + k][(R + r) * MB + m];
    }
    const size_t o = (size_t)(m0 + m) * N + n;
    if constexpr (DUAL) {
      if (use_bias) { v += to_f32<T>(bias0[n]); up += to_f32<T>(bias1[n]); }
      y[o] = from_f32<T>(silu(v) * up);
    } else {
      if (use_bias) v += to_f32<T>(bias0[n]);
      v = apply_act(v, activation);
      if (use_residual) v += to_f32<T>(residual[o]);
      y[o] = from_f32<T>(v);
    }
  }
}

template <int FMT, typename T, int MB, int R, bool DUAL>
static void launch_mb(cudaStream_t st, const GemvArgs& a) {
  const int steps = (int)((a.K + 255) / 256);
  const int64_t groups = (a.N + R - 1) / R;
  // warps share a row's steps until there are 24 warps per SM
  int slog = 0;
  while (slog < 3 && (groups << slog) < 24ll * sm_count() && (2 << slog) <= steps) ++slog;
  const int per_block = GEN_WARPS >> slog;
  const int vec = ((uintptr_t)a.x & (4 * sizeof(T) - 1)) == 0 && a.K % 4 == 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((groups + per_block - 1) / per_block), (unsigned)((a.M + MB - 1) / MB));
  cfg.blockDim = dim3(GEN_WARPS * 32);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, gemv_generic_kernel<FMT, T, MB, R, DUAL>, (const T*)a.x, (const uint8_t*)a.w0, (const uint8_t*)a.w1,
                     (const T*)a.bias0, (const T*)a.bias1, (const T*)a.residual, (T*)a.y, (int)a.M, (int)a.K, (int)a.N,
                     a.activation, a.use_bias, a.use_residual, slog, vec);
  note_launch();
}

template <int FMT, typename T, bool DUAL>
static void launch_fmt(cudaStream_t st, const GemvArgs& a) {
  constexpr int R = DUAL ? 2 : 4;                  // few activation rows: more weight rows in flight per lane
  if (a.M == 1) launch_mb<FMT, T, 1, R, DUAL>(st, a);
  else if (a.M == 2) launch_mb<FMT, T, 2, R, DUAL>(st, a);
  else if (a.M <= 4) launch_mb<FMT, T, 4, R / 2, DUAL>(st, a);
  else launch_mb<FMT, T, 8, R / 2, DUAL>(st, a);
}

template <typename T, bool DUAL>
static void launch_dtype(cudaStream_t st, const GemvArgs& a) {
  switch (a.format) {
    case F_Q4_0: launch_fmt<F_Q4_0, T, DUAL>(st, a); break;
    case F_Q8_0: launch_fmt<F_Q8_0, T, DUAL>(st, a); break;
    case F_Q6_K: launch_fmt<F_Q6_K, T, DUAL>(st, a); break;
    case F_MXFP8: launch_fmt<F_MXFP8, T, DUAL>(st, a); break;
    case F_NVFP4: launch_fmt<F_NVFP4, T, DUAL>(st, a); break;
    default: launch_fmt<F_MXFP4, T, DUAL>(st, a); break;
  }
}

void launch_gemv_generic(cudaStream_t st, const GemvArgs& a) {
  const bool dual = a.w1 != nullptr;
  if (a.dtype == QX_DTYPE_F32) {
    dual ? launch_dtype<float, true>(st, a) : launch_dtype<float, false>(st, a);
  } else if (a.dtype == QX_DTYPE_F16) {
    dual ? launch_dtype<__half, true>(st, a) : launch_dtype<__half, false>(st, a);
  } else {
    dual ? launch_dtype<__nv_bfloat16, true>(st, a) : launch_dtype<__nv_bfloat16, false>(st, a);
  }
}

}  // namespace qx
