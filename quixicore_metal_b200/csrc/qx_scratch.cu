// Host-side services shared by the entry points: device scratch for calls that bring no workspace,
// the tensor-map cache, and the path options.
#include <atomic>
#include <cstring>
#include <mutex>
#include <vector>

#include "qx_common.cuh"
#include "qx_kernels.h"
#include "qx_tmap.h"

namespace qx {

// ---- path options -----------------------------------------------------------------------------
static Options g_options;
const Options& options() { return g_options; }
bool set_option(const char* name, int value) {
  if (!name) return false;
  if (std::strcmp(name, "stream_passes") == 0 && value >= 0 && value <= 2) { g_options.stream_passes = value; return true; }
  if (std::strcmp(name, "force_generic") == 0) { g_options.force_generic = value != 0; return true; }
  if (std::strcmp(name, "tc_pipeline") == 0) { g_options.tc_pipeline = value != 0; return true; }
  if (std::strcmp(name, "ts_min_rows") == 0 && value >= 0) { g_options.ts_min_rows = value; return true; }
  if (std::strcmp(name, "lm_head_ksplit") == 0) { g_options.lm_head_ksplit = value != 0; return true; }
  return false;
}

// ---- library-managed scratch ------------------------------------------------------------------
// Used only when the caller passes no workspace.  Calls on one stream are ordered, so a buffer tied
// to (device, stream) can serve every call on that stream.  Up to 16 (device, stream) pairs get
// such a buffer.  It grows by allocating a larger one; the smaller one stays allocated until the
// process exits (work already enqueued may still read it), so growth never synchronises or frees:
// the total is below twice the largest request.  cudaStreamPerThread (one handle, a different
// stream in every thread), streams that are being captured, and pairs beyond the 16th take a
// stream-ordered allocation per call instead (*must_free: release with cudaFreeAsync on `st`).
struct ScratchSlot { int dev; cudaStream_t st; void* ptr; size_t bytes; };
static ScratchSlot g_scratch[16] = {};
static std::mutex g_scratch_mu;
static std::atomic<uint64_t> g_scratch_allocs{0};

uint64_t scratch_alloc_count() { return g_scratch_allocs.load(std::memory_order_relaxed); }

void* default_scratch(cudaStream_t st, size_t bytes, bool* must_free) {
  *must_free = false;
  if (bytes == 0) bytes = 256;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return nullptr; }
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) { cudaGetLastError(); cap = cudaStreamCaptureStatusNone; }
  if (cap == cudaStreamCaptureStatusNone && st != cudaStreamPerThread) {
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    ScratchSlot* slot = nullptr;
    for (auto& s : g_scratch) {
      if (s.ptr && s.dev == dev && s.st == st) { slot = &s; break; }
      if (!s.ptr && !slot) slot = &s;
    }
    if (slot && slot->ptr && slot->bytes >= bytes) return slot->ptr;
    if (slot) {
      size_t want = bytes < (1u << 20) ? (1u << 20) : bytes;
      if (slot->ptr && want < 2 * slot->bytes) want = 2 * slot->bytes;
      void* p = nullptr;
      if (cudaMalloc(&p, want) == cudaSuccess) {
        g_scratch_allocs.fetch_add(1, std::memory_order_relaxed);
        *slot = ScratchSlot{dev, st, p, want};      // a smaller predecessor stays allocated on purpose
        return p;
      }
      cudaGetLastError();
    }
  }
  void* p = nullptr;
  if (cudaMallocAsync(&p, bytes, st) != cudaSuccess) { cudaGetLastError(); return nullptr; }
  g_scratch_allocs.fetch_add(1, std::memory_order_relaxed);
  *must_free = true;
  return p;
}

// ---- tensor-map cache ---------------------------------------------------------------------------
// Encoding a tensor map is a driver call of a few microseconds; a decode loop calls the same weights
// every step.  Maps are cached per (device, base pointer, rows, row bytes, box).  A weight freed
// and another allocated at the same address with the same geometry yields the same map, so stale
// entries are harmless; the table is a small direct-mapped cache, collisions simply re-encode.
struct MapKey {
  int dev, elem_bytes, box_w, box_h; const void* base; int64_t width, height; size_t pitch;
  bool operator==(const MapKey& o) const {
    return dev == o.dev && elem_bytes == o.elem_bytes && box_w == o.box_w && box_h == o.box_h && base == o.base &&
           width == o.width && height == o.height && pitch == o.pitch;
  }
};
struct MapEntry { MapKey key; bool valid; CUtensorMap map; };
static MapEntry g_maps[1024];
static std::mutex g_maps_mu;

bool cached_box_map(CUtensorMap* map, const void* base, int elem_bytes, int64_t width, int64_t height, size_t pitch,
                    int box_w, int box_h) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return false; }
  const MapKey key{dev, elem_bytes, box_w, box_h, base, width, height, pitch};
  uint64_t h = (uint64_t)(uintptr_t)base * 0x9E3779B97F4A7C15ull;
  h ^= ((uint64_t)height * 31u + (uint64_t)box_w * 131u + (uint64_t)box_h * 8191u + (uint64_t)dev * 7u + (uint64_t)width) * 0xC2B2AE3D27D4EB4Full;
  MapEntry& e = g_maps[(h >> 40) & 1023u];
  {
    std::lock_guard<std::mutex> lock(g_maps_mu);
    if (e.valid && e.key == key) { *map = e.map; return true; }
  }
  TensorMapEncodeFn enc = tensor_map_encode_fn();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)height};
  const cuuint64_t strides[1] = {(cuuint64_t)pitch};
  const cuuint32_t box[2] = {(cuuint32_t)box_w, (cuuint32_t)box_h};
  const cuuint32_t estr[2] = {1u, 1u};
  if (enc(map, elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(base), dims,
          strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  std::lock_guard<std::mutex> lock(g_maps_mu);
  e = MapEntry{key, true, *map};
  return true;
}

bool cached_weight_map(CUtensorMap* map, const void* w, int64_t rows, size_t row_bytes, int box_bytes, int box_rows) {
  return cached_box_map(map, w, 4, (int64_t)(row_bytes / 4), rows, row_bytes, box_bytes / 4, box_rows);
}

}  // namespace qx
