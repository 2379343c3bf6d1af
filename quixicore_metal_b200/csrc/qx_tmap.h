// Host-side construction of the TMA tensor maps the kernels use for packed weight matrices.
#pragma once

#include <cstdint>

#include <cuda.h>
#include <cuda_runtime.h>

namespace qx {

// The driver entry point is looked up at run time, so the library does not link libcuda.
typedef CUresult (*TensorMapEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                      const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                      CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                      CUtensorMapFloatOOBfill);
inline TensorMapEncodeFn tensor_map_encode_fn() {
  static TensorMapEncodeFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      return (TensorMapEncodeFn) nullptr;
    }
    return (TensorMapEncodeFn)p;
  }();
  return fn;
}
// Tensor map over a packed weight matrix seen as rows of 32-bit words, box = (box_bytes / 4) words x
// box_rows rows; rows past the end read as zeros.  Through the cache of qx_scratch.cu.
bool cached_weight_map(CUtensorMap* map, const void* w, int64_t rows, size_t row_bytes, int box_bytes,
                       int box_rows = 128);

// General form: `height` rows of `width` elements of elem_bytes (2 or 4), `pitch` bytes apart, box_w x box_h elements.
bool cached_box_map(CUtensorMap* map, const void* base, int elem_bytes, int64_t width, int64_t height, size_t pitch,
                    int box_w, int box_h);

}  // namespace qx
