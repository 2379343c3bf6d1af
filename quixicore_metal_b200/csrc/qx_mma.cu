// decode_linear_epilogue / decode_swiglu for batch > 16 on the shared tcgen05 pipeline of qx_tc_pipeline.cuh (2-D TMA
// boxes of packed weights -> in-kernel dequant to f16 operand tiles -> tcgen05.mma, block scales applied from tensor
// memory): its projection epilogues (bias / activation / residual, the SwiGLU gate, raw fp32 partials) and the
// launch code.  Serves what qx_ts.cuh does not: K = 128 mod 256, and the ordered form of the post-scaled formats.
// Every wait on an mbarrier is bounded; on expiry the CTA raises the device error flag, stops
// issuing work, frees its tensor memory and returns.
#include "qx_kernels.h"
#include "qx_stream.cuh"
#include "qx_tc.cuh"
#include "qx_tc_pipeline.cuh"
#include "qx_tmap.h"

namespace qx {

// ---- projections on the shared tensor-core pipeline (qx_tc_pipeline.cuh) ---------------------------
// Epilogue: thread = one output channel n of the item, CW activation rows; 32 lanes store 32
// consecutive channels of one row.  Linear: y = act(v * rowscale + bias) (+ residual); an item is
// 256 channels.  SwiGLU: half 0 = gate rows, half 1 = up rows of the same 128 channels,
// y = silu(gate) * up.  Raw fp32 dot products when `raw` is set (row-parallel partials).
template <int BN, typename OT, bool DUAL_>
struct ProjEpi {
  struct Args {
    const OT* bias0; const OT* bias1; const OT* residual;
    void* y;
    int N, activation, use_bias, use_residual, raw;
    uint8_t* mx_blocks;     // fused MXFP8 output rows (N % 32 == 0): a warp holds one 32-channel block per row
  };
  static constexpr bool DUAL = DUAL_;
  __device__ __forceinline__ static bool packs_rows(const Args& a) { return a.mx_blocks != nullptr; }
  __device__ __forceinline__ static void run(const Args& a, const TcItem& it) {
    constexpr int CW = BN / 4;
    if (it.warp >= LTC_DQW) return;
    const uint32_t lane_sel = (uint32_t)((it.warp & 3) * 32) << 16;
    const int RS = (it.warp & 3) * 32 + it.lane;
    const int cg = it.warp >> 2;
    if constexpr (DUAL) {
      uint32_t g[CW], u[CW];
      tmem_ld_nowait<CW>(it.tmem_base + lane_sel + (uint32_t)(cg * CW), g);
      tmem_ld_nowait<CW>(it.tmem_base + lane_sel + (uint32_t)(BN + cg * CW), u);
      tmem_wait_ld();
      const int n = it.tile * 128 + RS;
      if (n < a.N) {
        const float gb = a.use_bias ? to_f32<OT>(a.bias0[n]) : 0.f;
        const float ub = a.use_bias ? to_f32<OT>(a.bias1[n]) : 0.f;
#pragma unroll
        for (int i = 0; i < CW; ++i) {
          const int m = cg * CW + i;
          if (m < it.m_count) {
            const float rs = it.rowscale[it.m_base + m];
            const float gv = __uint_as_float(g[i]) * rs + gb, uv = __uint_as_float(u[i]) * rs + ub;
            const OT out = from_f32<OT>(silu(gv) * uv);
            reinterpret_cast<OT*>(a.y)[(size_t)(it.m_base + m) * a.N + n] = out;
            if (a.mx_blocks)
              mxfp8_block_store(to_f32<OT>(out), it.lane,
                                a.mx_blocks + ((size_t)(it.m_base + m) * (a.N >> 5) + (n >> 5)) * 33);
          }
        }
      }
    } else {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t v[CW];
        tmem_ld_nowait<CW>(it.tmem_base + lane_sel + (uint32_t)(h * BN + cg * CW), v);
        tmem_wait_ld();
        const int n = it.tile * 256 + h * 128 + RS;
        if (n < a.N) {
          const float bv = (a.use_bias && !a.raw) ? to_f32<OT>(a.bias0[n]) : 0.f;
#pragma unroll
          for (int i = 0; i < CW; ++i) {
            const int m = cg * CW + i;
            if (m < it.m_count) {
              const size_t o = (size_t)(it.m_base + m) * a.N + n;
              const float dot = __uint_as_float(v[i]) * it.rowscale[it.m_base + m];
              if (a.raw) {
                reinterpret_cast<float*>(a.y)[o] = dot;
              } else {
                float val = apply_act(dot + bv, a.activation);
                if (a.use_residual) val += to_f32<OT>(a.residual[o]);
                const OT out = from_f32<OT>(val);
                reinterpret_cast<OT*>(a.y)[o] = out;
                if (a.mx_blocks)
                  mxfp8_block_store(to_f32<OT>(out), it.lane,
                                    a.mx_blocks + ((size_t)(it.m_base + m) * (a.N >> 5) + (n >> 5)) * 33);
              }
            }
          }
        }
      }
    }
  }
  __device__ __forceinline__ static void tail(const Args&, const float*, int, int, int) {}
};

template <int FMT, int BN, typename OT, bool DUAL>
static bool launch_pipeline_bn(cudaStream_t st, const GemvArgs& a, int* err) {
  using S = TcSmem<FMT, BN>;
  using C = TcCfg<FMT>;
  using Epi = ProjEpi<BN, OT, DUAL>;
  static_assert(S::TOTAL <= 227 * 1024, "tensor-core pipeline configuration exceeds shared memory");
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    if (cudaFuncSetAttribute(tc_pipeline_kernel<FMT, BN, Epi>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    attr_set[dev] = true;
  }
  const size_t row_bytes = (size_t)(a.K / StreamFmt<FMT>::BK) * StreamFmt<FMT>::BB;
  CUtensorMap map0, map1;
  if (!cached_weight_map(&map0, a.w0, a.N, row_bytes, C::BOX)) return false;
  if (DUAL) { if (!cached_weight_map(&map1, a.w1, a.N, row_bytes, C::BOX)) return false; }
  else map1 = map0;
  const int groups = (int)((a.M + BN - 1) / BN);
  const size_t img_bytes = ((size_t)groups * BN * a.K * 2 + 255) & ~(size_t)255;
  if (!a.scratch || a.scratch_bytes < img_bytes + (((size_t)a.M * 4 + 255) & ~(size_t)255)) return false;
  __half* ximg = (__half*)a.scratch;
  float* rowscale = (float*)((char*)a.scratch + img_bytes);
  if (!launch_prep_activations(st, a.x, a.dtype, ximg, rowscale, (int)a.M, (int)a.K, StreamFmt<FMT>::PERM, BN)) return false;
  const int item_rows = DUAL ? 128 : 256;
  const long long items = (long long)((a.N + item_rows - 1) / item_rows) * groups;
  const unsigned grid = (unsigned)(items < sm_count() ? items : sm_count());
  const typename Epi::Args ea{(const OT*)a.bias0, (const OT*)a.bias1, (const OT*)a.residual, a.y, (int)a.N,
                              a.activation, a.use_bias, a.use_residual, a.out_f32,
                              (a.out_quant == OQ_MXFP8 && !a.out_f32 && a.N % 32 == 0) ? (uint8_t*)a.q_codes : nullptr};
  tc_pipeline_kernel<FMT, BN, Epi><<<grid, LTC_WARPS * 32, S::TOTAL, st>>>(
      map0, map1, ximg, rowscale, (int)a.M, (int)a.N, (int)a.K, 1, err, ea);
  note_launch();
  return true;
}

template <int FMT, typename OT>
static bool launch_pipeline_fmt(cudaStream_t st, const GemvArgs& a, int* err) {
  if (a.w1) {
    if (a.M <= 32) return launch_pipeline_bn<FMT, 32, OT, true>(st, a, err);
    return launch_pipeline_bn<FMT, 64, OT, true>(st, a, err);
  }
  if (a.M <= 32) return launch_pipeline_bn<FMT, 32, OT, false>(st, a, err);
  return launch_pipeline_bn<FMT, 64, OT, false>(st, a, err);
}

// bf16 / f16 activations, batch > 16, 128-column multiples, 16-byte aligned rows, at least one
// full 128-row box; q6_K has no form here.
bool tc_path_ok(const GemvArgs& a) {
  if (a.dtype != QX_DTYPE_BF16 && a.dtype != QX_DTYPE_F16) return false;
  if (a.M <= 16 || a.format == F_Q6_K || a.K % 128 != 0 || a.N < 128) return false;
  const size_t row_bytes = (size_t)(a.K / block_k_of(a.format)) * block_bytes_of(a.format);
  if (row_bytes % 16 != 0 || ((uintptr_t)a.w0 & 15) != 0 || (a.w1 && ((uintptr_t)a.w1 & 15) != 0)) return false;
  return options().tc_pipeline;
}

// Scratch: the activation image + row scales.
size_t tc_scratch_bytes(const GemvArgs& a) {
  if (!tc_path_ok(a)) return 0;
  const int BN = a.M <= 32 ? 32 : 64;
  const size_t groups = (size_t)((a.M + BN - 1) / BN);
  return ((groups * BN * a.K * 2 + 255) & ~(size_t)255) + (((size_t)a.M * 4 + 255) & ~(size_t)255);
}

template <typename OT>
static bool launch_pipeline(cudaStream_t st, const GemvArgs& a, int* err) {
  switch (a.format) {
    case F_Q4_0: return launch_pipeline_fmt<F_Q4_0, OT>(st, a, err);
    case F_Q8_0: return launch_pipeline_fmt<F_Q8_0, OT>(st, a, err);
    case F_MXFP8: return launch_pipeline_fmt<F_MXFP8, OT>(st, a, err);
    case F_NVFP4: return launch_pipeline_fmt<F_NVFP4, OT>(st, a, err);
    case F_MXFP4: return launch_pipeline_fmt<F_MXFP4, OT>(st, a, err);
    default: return false;
  }
}

bool launch_gemm_tc(cudaStream_t st, const GemvArgs& a, bool* fused_quant) {
  int* err = device_error_flag();
  if (!err) return false;
  *fused_quant = true;
  return a.out_f32 ? launch_pipeline<float>(st, a, err)       // OT only types bias / residual, unused here
       : a.dtype == QX_DTYPE_F16 ? launch_pipeline<__half>(st, a, err)
                                 : launch_pipeline<__nv_bfloat16>(st, a, err);
}

}  // namespace qx
