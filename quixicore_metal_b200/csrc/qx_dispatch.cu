// Kernel-family selection for the projection ops.
#include "qx_common.cuh"
#include "qx_kernels.h"

namespace qx {

size_t projection_scratch_bytes(const GemvArgs& a) {
  if (options().force_generic) return 0;
  const size_t s = stream_scratch_bytes(a);
  size_t t = tc_scratch_bytes(a);
  if (t < s) t = s;
  const size_t u = ts_scratch_bytes(a);
  return t > u ? t : u;
}

// The tensor-core kernels, in order of preference; false when none serves the call.  *fused: the kernel
// also wrote the requested MXFP8 output rows.
bool launch_tensor_core(cudaStream_t st, const GemvArgs& a, bool* fused) {
  const bool fusable = a.out_quant == OQ_MXFP8 && !a.out_f32 && a.N % 32 == 0 && a.q_codes;
  *fused = false;
  if (options().force_generic) return false;
  // all of them read the activations in 16-byte vectors; ones that start elsewhere take the generic kernel
  if (((uintptr_t)a.x & 15) != 0) return false;
  const bool passes_first = options().stream_passes == 2 && stream_passes_ok(a);
  if (!passes_first && launch_ts(st, a, fused)) return true;
  *fused = fusable;
  if (stream_path_ok(a) && launch_gemv_stream(st, a)) return true;
  if (stream_passes_ok(a) && launch_gemv_stream_passes(st, a)) return true;
  if (tc_path_ok(a) && launch_gemm_tc(st, a, fused)) { *fused = fusable && *fused; return true; }
  *fused = false;
  return false;
}

// Returns true when the kernel that ran also wrote the requested MXFP8 output rows; every other
// output quantisation is a second launch by the caller.
bool launch_projection(cudaStream_t st, const GemvArgs& a) {
  bool fused = false;
  if (launch_tensor_core(st, a, &fused)) return fused;
  launch_gemv_generic(st, a);
  return false;
}

}  // namespace qx
