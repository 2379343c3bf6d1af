// Activation preparation of every tensor-core path: a row of 16-bit activations -> f16 scaled by a power of two, its
// columns in the order and its 16-byte chunks at the places that the consuming kernel reads.
#include "qx_kernels.h"
#include "qx_stream.cuh"
#include "qx_ts.cuh"

namespace qx {

// Where a chunk of 8 prepared columns comes from and goes to.  Chunk c (0 .. 3) of a 32-column unit holds the columns
// from (c >> 1) * a + (c & 1) * b, four there and four `d` further: pairs w0 w1 | w2 w3.  The orders differ in how the
// pairs are mixed: words (x0, x1) and (x2, x3) through the byte selectors lo and hi, w1 and w2 exchanged before or the
// two middle words after.  Chunk i of the row lands at (i >> 3) * s1 + ((i & 7) ^ (row & swz)) * s2 behind its row's
// start, group * group_step + row * row_step (16-byte units), `rows` rows to a group.
struct PrepLayout {
  int a, b, d;
  uint32_t lo, hi;
  int swap_in, swap_out;
  int rows, row_step, s1, s2, swz;
  long long group_step;
};

// One CTA per row.  Largest finite magnitude -> scale 2^-S that puts it in [2^14, 2^15), then f16(x * 2^-S).  Bound by
// latencies: the launch, one read of a row from memory, and the code itself, which the weight stream of every call pushes
// out of L2.  So one copy of it serves all orders (orders as compile-time branches with 2-byte reads held the
// contraction's start up by 13 us of a 58 us call, nvfp4, 32 rows, K = 8192).
template <typename T>
__global__ void __launch_bounds__(512)
prep_rows_kernel(const T* __restrict__ x, uint4* __restrict__ out, float* __restrict__ rowscale, unsigned* __restrict__ count,
                 int ncount, int M, int K, const PrepLayout L) {
  __shared__ uint32_t red[16];
  // First the wait: the contraction may be scheduled once every CTA is past it, so all that ran before this kernel is
  // complete then - its weight loads need no wait of their own (an earlier kernel of the stream may have written
  // them), and its bounded waits do not count while a long predecessor runs.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  constexpr bool BF = sizeof(T) == 2 && std::is_same<T, __nv_bfloat16>::value;
  constexpr uint32_t MOST = BF ? 0x7F61u : 0x7BFFu;                    // largest magnitude (bits) that may choose the scale
  const int m = blockIdx.x, chunks = K >> 3, tid = threadIdx.x, step = blockDim.x;   // (a multiple of 32)
  const bool real = m < M;                                             // else a row of zeros that fills up a group
  if (m == 0)
#pragma unroll 1
    for (int i = tid; i < ncount; i += step) count[i] = 0u;
  // this thread's chunks are tid, tid + step, ..: all at the same place of their unit
  const uint2* src = reinterpret_cast<const uint2*>(x + (size_t)(real ? m : 0) * K) + (tid >> 2) * 8 + (((tid & 3) >> 1) * L.a + (tid & 1) * L.b) / 4;
  uint2 p[2], q[2];                                                    // the first two are kept, the others read again
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const bool in = real && tid + r * step < chunks;
    p[r] = in ? __ldg(src + r * step * 2) : make_uint2(0u, 0u);
    q[r] = in ? __ldg(src + r * step * 2 + L.d / 4) : make_uint2(0u, 0u);
  }
  uint32_t most = 0u;                                                  // largest magnitudes of both halves side by side
  auto fold = [&](uint2 v) { most = __vmaxu2(most, __vmaxu2(v.x & 0x7FFF7FFFu, v.y & 0x7FFF7FFFu)); };
  fold(p[0]); fold(q[0]); fold(p[1]); fold(q[1]);
  if (real)
#pragma unroll 1
    for (int i = tid + 2 * step, o = 4 * step; i < chunks; i += step, o += 2 * step) { fold(__ldg(src + o)); fold(__ldg(src + o + L.d / 4)); }
  auto reduce = [&](uint32_t v) {
    v = __reduce_max_sync(0xffffffffu, v);
    if ((tid & 31) == 0) red[tid >> 5] = v;
    __syncthreads();
    return __reduce_max_sync(0xffffffffu, (tid & 31) < (step >> 5) ? red[tid & 31] : 0u);
  };
  uint32_t top = reduce(max(most & 0xFFFFu, most >> 16));
  if (top > MOST) {                                                    // infinities, NaN and bf16 from 3e38 do not choose the scale
    most = 0u;
#pragma unroll 1
    for (int i = tid; i < K; i += step) {
      const uint32_t v = __ldg(reinterpret_cast<const uint16_t*>(x) + (size_t)m * K + i) & 0x7FFFu;
      if (v <= MOST) most = max(most, v);
    }
    __syncthreads();
    top = reduce(most);
  }
  int S = 0;
  if (top != 0u) {
    const float amax = BF ? __uint_as_float(top << 16) : __half2float(__ushort_as_half((unsigned short)top));
    S = (int)((__float_as_uint(amax) >> 23) & 0xFFu) - 127 - 14;
    S = max(-110, min(110, S));
  }
  const float down = __uint_as_float((uint32_t)(127 - S) << 23);       // 2^-S
  const int grp = m / L.rows, ml = m - grp * L.rows;
  uint4* o = out + (size_t)grp * L.group_step + (size_t)ml * L.row_step + (size_t)(tid >> 3) * L.s1 + ((tid & 7) ^ (ml & L.swz)) * L.s2;
  auto half2 = [&](uint32_t w) {
    float2 f;
    if constexpr (BF) f = make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
    else f = __half22float2(*reinterpret_cast<const __half2*>(&w));
    const __half2 h = __floats2half2_rn(f.x * down, f.y * down);
    return *reinterpret_cast<const uint32_t*>(&h);
  };
#pragma unroll 1
  for (int i = tid, r = 0; i < chunks; i += step, ++r, src += step * 2, o += (size_t)(step >> 3) * L.s1) {
    if (r >= 2 && real) { p[0] = __ldg(src); q[0] = __ldg(src + L.d / 4); }
    const uint32_t w0 = half2(p[0].x), w1 = half2(p[0].y), w2 = half2(q[0].x), w3 = half2(q[0].y);
    const uint32_t x1 = L.swap_in ? w2 : w1, x2 = L.swap_in ? w1 : w2;
    const uint32_t o1 = __byte_perm(w0, x1, L.hi), o2 = __byte_perm(x2, w3, L.lo);
    *o = make_uint4(__byte_perm(w0, x1, L.lo), L.swap_out ? o2 : o1, L.swap_out ? o1 : o2, __byte_perm(x2, w3, L.hi));
    p[0] = p[1]; q[0] = q[1];
  }
  if (tid == 0 && real) rowscale[m] = __uint_as_float((uint32_t)(127 + S) << 23);
}

static bool launch_prep(cudaStream_t st, const void* x, qx_dtype dtype, void* out, float* rowscale, unsigned* count, int ncount,
                        int M, int rows, int K, const PrepLayout& L) {
  const dim3 block(K >= 4096 ? 512 : 256);
  if (dtype == QX_DTYPE_F16)
    return ts_launch_dependent(st, dim3(rows), block, 0, prep_rows_kernel<__half>, (const __half*)x, (uint4*)out, rowscale, count, ncount, M, K, L);
  return ts_launch_dependent(st, dim3(rows), block, 0, prep_rows_kernel<__nv_bfloat16>, (const __nv_bfloat16*)x, (uint4*)out, rowscale, count, ncount, M, K, L);
}

// The orders of perm_position (1 .. 5, 0 = as they are).
static PrepLayout perm_layout(int perm) {
  PrepLayout L{};
  L.lo = 0x5410; L.hi = 0x7632;
  switch (perm) {
    case 1: L.a = 8;  L.b = 4; L.d = 16; break;                                  // a0 a2 a1 a3 b0 b2 b1 b3
    case 2: L.a = 8;  L.b = 4; L.d = 16; L.swap_in = 1; break;                   // a0 b0 a1 b1 a2 b2 a3 b3
    case 3: L.a = 16; L.b = 4; L.d = 8;  L.swap_in = 1; break;
    case 4: L.a = 16; L.b = 8; L.d = 4;  break;
    case 5: L.a = 16; L.b = 8; L.d = 4;  L.swap_in = 1; break;
    default: L.a = 16; L.b = 8; L.d = 4; L.lo = 0x3210; L.hi = 0x7654;
  }
  return L;
}

// img_rows > 0: the operand-tile image that the tcgen05 pipeline copies in bulk, else plain rows.  Rows are taken in
// groups of img_rows; a group is stored k-stage by k-stage (64 columns = 128 bytes per row), each stage as img_rows
// consecutive 128-byte rows whose 16-byte chunks are XOR-swizzled with the row index (the 128-byte swizzle of a K-major
// operand tile); rows past M are zero.
bool launch_prep_activations(cudaStream_t st, const void* x, qx_dtype dtype, __half* x16, float* rowscale, int M, int K, int perm,
                             int img_rows) {
  PrepLayout L = perm_layout(perm);
  L.s2 = 1;
  int rows = M;
  if (img_rows > 0) {
    L.rows = img_rows; L.group_step = (long long)img_rows * (K / 8); L.row_step = 8; L.s1 = 8 * img_rows; L.swz = 7;
    rows = (M + img_rows - 1) / img_rows * img_rows;
  } else {
    L.rows = 1; L.group_step = K / 8; L.s1 = 8;
  }
  return launch_prep(st, x, dtype, x16, rowscale, nullptr, 0, M, rows, K, L);
}

// The image [group][K / 8][mp][8] of the tensor-memory-operand kernel (16-byte chunks of one row, mp rows side by side:
// the unswizzled operand layout), 32-column units in the order of ts_position; its tickets are zeroed too.  Rows past a
// group's end are never read back.
bool ts_launch_prep(cudaStream_t st, const TsPlan& p, int format, const void* x, qx_dtype dtype, const TsScratch& s, int M, int K) {
  PrepLayout L = perm_layout(format == F_MXFP4 ? 2 : (format == F_NVFP4 ? 3 : (format == F_Q4_0 ? 1 : 0)));
  if (format == F_Q4_0) L.swap_out = 1;                                          // a0 a2 b0 b2 a1 a3 b1 b3
  L.rows = p.mg; L.group_step = (long long)(K / 8) * p.mp; L.row_step = 1; L.s1 = 8 * p.mp; L.s2 = p.mp;
  return launch_prep(st, x, dtype, s.img, s.rowscale, s.count, p.whole ? 0 : p.items, M, M, K, L);
}

}  // namespace qx
