// Host side and projection epilogue of the tensor-memory-operand kernel (qx_ts.cuh): plans, tensor maps, the rule that
// chooses it, and the launches behind decode_linear_epilogue / decode_swiglu.
#include "qx_kernels.h"
#include "qx_tmap.h"
#include "qx_ts.cuh"

namespace qx {

static size_t round256(size_t n) { return (n + 255) & ~(size_t)255; }

struct TsGeom { int bytes, pitch, terms; };
static TsGeom ts_geom(int f) {
  switch (f) {
    case F_Q4_0: return {TsFmt<F_Q4_0>::BYTES, TsFmt<F_Q4_0>::PITCH, TsFmt<F_Q4_0>::TERMS};
    case F_Q8_0: return {TsFmt<F_Q8_0>::BYTES, TsFmt<F_Q8_0>::PITCH, TsFmt<F_Q8_0>::TERMS};
    case F_Q6_K: return {TsFmt<F_Q6_K>::BYTES, TsFmt<F_Q6_K>::PITCH, TsFmt<F_Q6_K>::TERMS};
    case F_MXFP8: return {TsFmt<F_MXFP8>::BYTES, TsFmt<F_MXFP8>::PITCH, TsFmt<F_MXFP8>::TERMS};
    case F_NVFP4: return {TsFmt<F_NVFP4>::BYTES, TsFmt<F_NVFP4>::PITCH, TsFmt<F_NVFP4>::TERMS};
    default: return {TsFmt<F_MXFP4>::BYTES, TsFmt<F_MXFP4>::PITCH, TsFmt<F_MXFP4>::TERMS};
  }
}

// K in whole raw stages (so every row is a multiple of 8 bytes; q6_K of 2), 16-byte aligned matrices.
bool ts_shape_ok(int format, int64_t K, int64_t N, const void* w0, const void* w1) {
  return K % TS_KC == 0 && N >= 8 && (((uintptr_t)w0 | (uintptr_t)w1) & 15) == 0;
}

bool ts_plan(TsPlan* p, int format, int64_t M, int64_t K, int64_t N, int rb, int dual, int max_group, size_t aux, bool may_cut) {
  const TsGeom g = ts_geom(format);
  const int64_t row_bytes = K / TS_KC * g.bytes;
  p->dual = dual; p->rb = dual ? 2 : rb;
  p->P = 1;
  while ((row_bytes * p->P) % 16 != 0) p->P *= 2;
  p->groups = (int)((M + max_group - 1) / max_group);
  p->mg = (int)((M + p->groups - 1) / p->groups);
  p->nb = (p->mg + 15) / 16 * 16;
  p->mp = p->mg <= 1 ? 1 : (p->mg <= 2 ? 2 : (p->mg <= 4 ? 4 : (p->mg <= 8 ? 8 : p->nb)));
  p->tile_rows = dual ? 128 : 128 * rb;
  p->tiles = (int)((N + p->tile_rows - 1) / p->tile_rows);
  p->nks = (int)(K / TS_KC);
  p->items = p->tiles * p->groups;
  // TMEM (512 columns): running sums and two chunk buffers of rb * nb columns, the rest operand slots, at least
  // one per worker group (so that a group's waits are never two ring rounds apart).  With two row blocks one chunk
  // buffer is enough: the blocks take turns.  Without room for the sums (128 rows and two blocks) an
  // item is one chunk - a format whose terms are short enough for that only (max_group).
  const int slot = 32 * g.terms, acc = p->rb * p->nb, least = 4 * slot;
  p->sums = 1;
  if (3 * acc + 2 * least <= 512) p->nd = 2;
  else if (p->rb == 2 && 2 * acc + 2 * least <= 512) p->nd = 1;      // eight slots (two issuers) before a second buffer
  else if (3 * acc + least <= 512) p->nd = 2;
  else if (2 * acc + least <= 512) p->nd = 1;
  else if (acc + least <= 512) { p->sums = 0; p->nd = 1; }
  else return false;
  p->na = (512 - (p->sums + p->nd) * acc) / slot;
  p->na = p->na >= 16 && format != F_Q6_K ? 16 : (p->na >= 8 && format != F_Q6_K ? 8 : 4);
  p->issuers = p->rb == 2 && p->na >= 8 ? 2 : 1;
  // Activation stages of 256 columns: at least two, and the raw ring takes the rest.  (One of 128 rows, handed over by
  // quarters beside a longer raw ring, costs the issuers a wait per quarter: 8192 -> 28672, mxfp4, 256 rows, 190 us
  // against 186; 4096 -> 14336, nvfp4, 128 rows, 53.5 against 49.5.)
  const size_t act_stage = (size_t)TS_KC * p->mp * 2;
  p->nact = p->mp <= 16 ? 4 : (p->mp <= 32 ? 3 : 2);
  const size_t stage = (size_t)128 * g.pitch;
  const size_t bar_bytes = 8 * (2 * TS_MAX_RAW + 2 * TS_MAX_ACT + 2 * TS_MAX_SLOTS + 12) + 4 * (4 + TS_MARK_RING * 8 + 128 + 256);
  const size_t act = (act_stage * p->nact + 256 + 127) & ~(size_t)127;   // + what overlapping core matrices read past the end
  const size_t fixed = act + ((aux + 127) & ~(size_t)127) + bar_bytes + 128;
  if (fixed + 2 * stage > 227 * 1024) return false;
  p->nraw = (int)((227 * 1024 - fixed) / stage);
  if (p->nraw > TS_MAX_RAW) p->nraw = TS_MAX_RAW;
  if (format == F_Q6_K) p->nraw &= ~1;               // its worker groups alternate stages: a slot always has the same readers
  p->off_act = stage * p->nraw;
  p->off_aux = p->off_act + act;
  p->off_bar = p->off_aux + ((aux + 127) & ~(size_t)127);
  p->smem = p->off_bar + bar_bytes + 128;
  // grid: every SM, a multiple of the groups, no CTA without a unit
  const int sms = sm_count();
  if (p->groups > sms || (int64_t)p->tiles * p->nks >= (1 << 30)) return false;
  p->whole = may_cut ? 0 : 1;
  const int64_t units = may_cut ? (int64_t)p->tiles * p->nks : p->tiles;
  const int64_t per = sms / p->groups;
  p->grid = (unsigned)((per < units ? per : units) * p->groups);
  p->img_bytes = round256((size_t)p->groups * p->mp * K * 2);
  p->scale_bytes = round256((size_t)M * 4);
  p->count_bytes = may_cut ? round256((size_t)p->items * 4) : 0;
  p->part_bytes = (size_t)p->grid * 4 * p->rb * p->nb * 128 * 4;
  return true;
}

TsScratch ts_carve(const TsPlan& p, void* scratch) {
  char* c = (char*)scratch;
  TsScratch s;
  s.img = (uint8_t*)c;
  s.rowscale = (float*)(c + p.img_bytes);
  s.count = (unsigned*)(c + p.img_bytes + p.scale_bytes);
  s.part = (float*)(c + p.img_bytes + p.scale_bytes + p.count_bytes);
  return s;
}

bool ts_maps(const TsPlan& p, int format, const void* w, int64_t K, int64_t N, CUtensorMap* m) {
  const TsGeom g = ts_geom(format);
  const int64_t row_bytes = K / TS_KC * g.bytes;
  if (p.P == 1) {
    if (!cached_box_map(&m[0], w, 4, row_bytes / 4, N, (size_t)row_bytes, g.pitch / 4, 128)) return false;
    m[1] = m[0];
    return true;
  }
  const int64_t full = N / p.P, rest = N % p.P;
  const size_t pitch = (size_t)(row_bytes * p.P);
  if (!cached_box_map(&m[1], w, 2, row_bytes * p.P / 2, full, pitch, g.pitch / 2, 128 / p.P)) return false;
  m[0] = m[1];
  // the last, partial super-row holds `rest` rows: nothing past the matrix may be touched
  return rest == 0 || cached_box_map(&m[0], w, 2, row_bytes * rest / 2, full + 1, pitch, g.pitch / 2, 128 / p.P);
}

// ---- projection epilogue ------------------------------------------------------------------------------
struct TsProj {
  struct Args {
    const void* bias0; const void* bias1; const void* residual; void* y;
    int half;                 // I/O type: 1 f16, 0 bf16 (bias, residual, output)
    int raw;                  // output fp32 dots, nothing else applied
    int activation, use_bias, use_residual;
    uint8_t* mx;              // MXFP8 rows of the rounded output (N % 32 == 0)
  };
  __device__ __forceinline__ static bool packs_rows(const Args& a) { return a.mx != nullptr; }
  __device__ __forceinline__ static float load(const void* p, size_t i, int half) {
    const uint16_t b = reinterpret_cast<const uint16_t*>(p)[i];
    return half ? __half2float(__ushort_as_half(b)) : __uint_as_float((uint32_t)b << 16);
  }
  static constexpr int AUX = 0;
  static constexpr bool HELP = true;
  // Eight columns at a time: warps w, w + 4, .. take the groups of eight in turn, a lane one weight row.  The reads of a
  // group are in flight together, then every step runs over all eight (with one column after the other, four reads
  // ahead, an item of 256 x 128 took 110,000 clocks, most of them one warp's latencies).  MXFP8 rows are packed from
  // the registers (a block is 32 lanes): in a second pass over y they cost 128 us of 272 at 256 x 28672.
  static constexpr int COLS = 8;
  __device__ __forceinline__ static void sum(const TsItem& it, size_t at, float (&v)[COLS]) {
#pragma unroll
    for (int i = 0; i < COLS; ++i) v[i] = __ldcg(it.first + at + i * 128);
#pragma unroll 1
    for (int k = 1; k < it.parts; ++k) {
      const float* s = it.part(k) + at;
#pragma unroll
      for (int i = 0; i < COLS; ++i) v[i] += __ldcg(s + i * 128);
    }
  }
  template <bool SHIFT>
  __device__ __forceinline__ static void run(const Args& a, const TsParams& q, const TsItem& it, const float* scale, const float* back,
                                             uint8_t*, int warp, int warps, int lane) {
    const TsPlan& p = q.p;
    const int blocks = p.dual ? 1 : p.rb;
    const int row = (warp & 3) * 32 + lane;
#pragma unroll 1
    for (int rb = 0; rb < blocks; ++rb) {
      const int n = it.tile * p.tile_rows + rb * 128 + row;
      if (n >= q.N) continue;
      const float b0 = a.use_bias ? load(a.bias0, n, a.half) : 0.f;
      const float b1 = p.dual && a.use_bias ? load(a.bias1, n, a.half) : 0.f;
#pragma unroll 1
      for (int c = (warp >> 2) * COLS; c < it.m_count; c += (warps >> 2) * COLS) {
        const int cols = it.m_count - c;                             // (columns past the group: read, not written)
        const size_t o = (size_t)(it.m_base + c) * q.N + n;
        float v[COLS], w[COLS];
        if (a.use_residual) {
#pragma unroll
          for (int i = 0; i < COLS; ++i) w[i] = i < cols ? load(a.residual, o + (size_t)i * q.N, a.half) : 0.f;
        }
        sum(it, ((size_t)rb * p.nb + c) * 128 + row, v);
        if (p.dual) sum(it, ((size_t)p.nb + c) * 128 + row, w);
        const float f0 = SHIFT ? back[rb * 128 + row] : 1.f;
#pragma unroll
        for (int i = 0; i < COLS; ++i) v[i] = SHIFT ? v[i] * scale[c + i] * f0 : v[i] * scale[c + i];
        if (a.raw) {
#pragma unroll
          for (int i = 0; i < COLS; ++i)
            if (i < cols) reinterpret_cast<float*>(a.y)[o + (size_t)i * q.N] = v[i];
          continue;
        }
        if (p.dual) {
          const float f1 = SHIFT ? back[128 + row] : 1.f;
#pragma unroll
          for (int i = 0; i < COLS; ++i) {
            const float u = SHIFT ? w[i] * scale[c + i] * f1 : w[i] * scale[c + i];
            v[i] = silu(v[i] + b0) * (u + b1);
          }
        } else {
#pragma unroll
          for (int i = 0; i < COLS; ++i) v[i] += b0;
          if (a.activation == 2) {
#pragma unroll
            for (int i = 0; i < COLS; ++i) v[i] = silu(v[i]);
          } else if (a.activation == 1) {
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {                            // (four copies of its code, not eight)
              float t[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) { t[i] = gelu_erf_as(v[i]); v[i] = v[i + 4]; }
#pragma unroll
              for (int i = 0; i < 4; ++i) v[i + 4] = t[i];
            }
          }
          if (a.use_residual) {
#pragma unroll
            for (int i = 0; i < COLS; ++i) v[i] += w[i];
          }
        }
#pragma unroll
        for (int i = 0; i < COLS; ++i) {
          const uint16_t h = a.half ? __half_as_ushort(__float2half_rn(v[i])) : __bfloat16_as_ushort(__float2bfloat16_rn(v[i]));
          if (i < cols) reinterpret_cast<uint16_t*>(a.y)[o + (size_t)i * q.N] = h;
          v[i] = a.half ? __half2float(__ushort_as_half(h)) : __uint_as_float((uint32_t)h << 16);
        }
        if (a.mx) {                                                  // N % 32 == 0: 32 lanes = 32 consecutive channels
          uint8_t* blk = a.mx + ((size_t)(it.m_base + c) * (q.N >> 5) + (n >> 5)) * 33;
#pragma unroll
          for (int i = 0; i < COLS; ++i)
            if (i < cols) mxfp8_block_store(v[i], lane, blk + (size_t)i * (q.N >> 5) * 33);
        }
      }
    }
  }
  __device__ __forceinline__ static void tail(const Args&, const TsParams&, uint8_t*, int, int) {}
};

// Row blocks per item: two share every activation stage (half the L2 reads of the activations) while there
// are enough of them to keep the cut items few.
static int ts_blocks(const GemvArgs& a) { return a.N >= 128 * 148 ? 2 : 1; }

// Row groups of one launch (4 CTAs each on 148 SMs); more rows take several launches.
constexpr int64_t TS_PASS_GROUPS = 37;

// Activation rows per group: 64 with running sums; nvfp4 and mxfp4, whose products have at most 14 bits, take 128 in
// one chunk per item (error at K = 8192: 1e-6 and 4e-7), which decodes the weights half as often.
static bool ts_projection_plan(const GemvArgs& a, TsPlan* p) {
  if (a.dtype != QX_DTYPE_BF16 && a.dtype != QX_DTYPE_F16) return false;
  if (((uintptr_t)a.x & 15) != 0 || !ts_shape_ok(a.format, a.K, a.N, a.w0, a.w1)) return false;
  const bool short_terms = a.format == F_NVFP4 || a.format == F_MXFP4;
  const int rb = a.format == F_Q6_K && a.M > 32 && !a.w1 ? 1 : ts_blocks(a);
  const int group = a.format == F_Q6_K ? (a.w1 ? 32 : 64) : (short_terms ? 128 : 64);
  const int64_t M = a.M < TS_PASS_GROUPS * group ? a.M : TS_PASS_GROUPS * group;
  if (!a.ordered) return ts_plan(p, a.format, M, a.K, a.N, rb, a.w1 != nullptr, group, 0, true);
  // A fixed order: items whole.  nvfp4 in the one accumulator over the whole of K of the in-place pipeline, whose
  // sums it continues; the other formats, which have no such form here, keep rounded sums over chunks (q6_K, K = 27648: one
  // accumulator over 5184 truncating steps is 1e-4 too small).
  if (!ts_plan(p, a.format, M, a.K, a.N, rb, a.w1 != nullptr, group, 0, false)) return false;
  if (a.format == F_NVFP4) p->sums = 0;
  return true;
}

// Where this kernel takes over from the 16-row streaming kernel (and its passes).  Its time hardly depends on the rows (and
// little on the bytes), the other's grows with them, fastest for the formats that cost most to decode.  us, streaming / this
// kernel:          4096 -> 4096   4096 -> 14336  8192 -> 28672
//   nvfp4  9 rows    10.3 / 14.9    19.4 / 21.5    47.6 / 40.2
//         16         11.4 / 15.1    21.0 / 21.5    51.7 / 40.4
//         32         15.0 / 15.8    29.8 / 22.0   100.8 / 41.5
//   mxfp4  9         11.9 / 16.1    22.7 / 22.5    64.9 / 46.9
//         16         13.0 / 16.3    26.7 / 22.7    72.9 / 46.9
//   mxfp8  9         14.4 / 19.1    30.0 / 29.7    91.0 / 72.6
//   q4_0   9         11.4 / 16.5    21.9 / 25.3    57.7 / 60.3
//         16         11.8 / 16.8    23.4 / 25.4    61.2 / 60.2
//         17         14.6 / 17.1    28.8 / 26.0   137.6 / 61.8
//   q8_0   9         12.2 / 18.0    21.1 / 27.1    57.3 / 63.9
//         16         13.3 / 18.0    24.5 / 27.2    73.6 / 64.0
//   q6_K  16         15.4 / 22.8    32.7 / 42.6   102.7 / 123.8
//         17         17.4 / 23.1    34.8 / 43.4   118.9 / 126.6
//         32         23.7 / 23.3    54.2 / 43.7   201.3 / 127.1
// At the lines: mxfp4 28 MiB, 12 / 16 rows 22.9 / 23.7 and 24.1 / 23.7, 56 MiB, 9 rows 33.2 / 31.2; nvfp4 64 MiB, 12 / 16 rows
// 30.0 / 31.2 and 32.6 / 31.1, 100 MiB, 9 rows 38.8 / 35.8; mxfp8 56 MiB, 9 / 16 rows 28.5 / 29.8 and 31.1 / 30.1; q8_0 189 MiB,
// 12 / 16 rows 49.5 / 56.3 and 54.4 / 56.3, 238 MiB, 12 rows 64.3 / 64.0; from 17 rows 28 MiB nvfp4 23.1 / 21.9, mxfp4 24.7 / 23.1,
// q4_0 26.3 / 26.3, q8_0 18.7 / 20.7 (34 MiB 22.4 / 22.4), mxfp8 20.9 / 22.4 (33 MiB 24.9 / 23.5); q6_K 20 / 22 rows, 46 MiB
// 38.9 / 43.0 and 42.9 / 43.1, 92 MiB 66.4 / 71.8 and 72.3 / 71.9 (28 MiB cross at 27 rows, 184 MiB at 19).
// SwiGLU pairs (bytes of both matrices), 9 and 16 rows, then 17 and 32 rows in 16-row passes:
//   nvfp4   63 MiB  27.3 / 27.4, 28.8 / 26.6;  45.5 / 27.8, 55.1 / 27.5     100 MiB  34.9 / 35.4, 36.8 / 34.7
//   mxfp4   68      30.6 / 34.5, 33.4 / 33.8                                119      50.2 / 46.7, 53.9 / 46.1
//   mxfp8   74      30.4 / 34.3, 31.6 / 33.4                                116      44.9 / 45.3, 46.6 / 44.1
//   q4_0   126      51.4 / 59.9, 52.3 / 59.0;  84.7 / 62.0, 102.9 / 61.8    252      86.8 / 101.4, 88.9 / 100.5
//   q8_0   238      55.8 / 64.0, 62.2 / 63.6; 107.5 / 66.2, 129.4 / 68.8    476      97.9 / 111.7, 110.3 / 113.8
//   q6_K   184      74.5 / 123, 91.6 / 123;    149 / 126, 182 / 127
//   16 MiB, 17 and 32 rows: nvfp4 22.4 / 19.6, 28.1 / 19.0; q4_0 23.3 / 23.9, 28.7 / 24.7; q8_0 20.6 / 23.0, 23.6 / 22.4
// Rows whose byte pitch the streaming kernel cannot take come here at every batch (the alternative is the scalar kernel: mxfp8
// K = 1280, 15 rows, gate / up / down of 5888: 512 us).
bool ts_preferred(const GemvArgs& a) {
  const int first = options().ts_min_rows;
  if (first > 0) return a.M >= first;
  const int64_t bytes = a.N * (a.K / block_k_of(a.format)) * block_bytes_of(a.format) * (a.w1 ? 2 : 1);
  if (a.ordered)                    // nvfp4: the pipeline's sums, bit for bit; and what no other kernel takes above 16 rows
    return a.M > 16 && !stream_passes_ok(a) && (a.format == F_NVFP4 || !tc_path_ok(a));
  if (a.M > 32) return true;
  if (!stream_path_ok(a) && !stream_passes_ok(a)) return true;
  if (a.M > 16) return bytes >= (a.w1 ? (16 << 20) : (28 << 20)) && !(a.format == F_Q6_K && !a.w1 && a.M <= 20);
  if (a.M <= 8) return false;
  const bool many = a.M >= 12;
  switch (a.format) {
    case F_NVFP4: return bytes >= (many && !a.w1 ? (64 << 20) : (100 << 20));
    case F_MXFP4: return bytes >= (a.w1 ? (100 << 20) : (many ? (28 << 20) : (56 << 20)));
    case F_MXFP8: return bytes >= (a.w1 ? (100 << 20) : (56 << 20));
    case F_Q8_0: return many && !a.w1 && bytes >= (200 << 20);
    default: return false;
  }
}

size_t ts_scratch_bytes(const GemvArgs& a) {
  TsPlan p;
  return ts_preferred(a) && ts_projection_plan(a, &p) ? p.scratch() : 0;
}

template <int FMT>
static bool launch_ts_fmt(cudaStream_t st, const GemvArgs& a, const TsPlan& p, int* err, bool* fused) {
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return false;
  if (!attr_set[dev]) {
    if (cudaFuncSetAttribute(ts_kernel<FMT, TsProj>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    attr_set[dev] = true;
  }
  CUtensorMap m[4];
  if (!ts_maps(p, FMT, a.w0, a.K, a.N, m)) return false;
  if (a.w1) { if (!ts_maps(p, FMT, a.w1, a.K, a.N, m + 2)) return false; }
  else { m[2] = m[0]; m[3] = m[1]; }
  const TsScratch s = ts_carve(p, a.scratch);
  TsParams q{p, {(const uint8_t*)a.w0, (const uint8_t*)a.w1}, a.x, a.dtype == QX_DTYPE_BF16, s.img, s.rowscale, s.part, s.count,
             (int)a.M, (int)a.K, (int)a.N, err};
  *fused = a.out_quant == OQ_MXFP8 && !a.out_f32 && a.N % 32 == 0 && a.q_codes;
  const TsProj::Args ea{a.bias0, a.bias1, a.residual, a.y, a.dtype == QX_DTYPE_F16, a.out_f32, a.activation, a.use_bias,
                        a.use_residual, *fused ? (uint8_t*)a.q_codes : nullptr};
  return ts_launch_prep(st, p, FMT, a.x, a.dtype, s, (int)a.M, (int)a.K) &&
         ts_launch_dependent(st, dim3(p.grid), dim3(TS_WARPS * 32), p.smem, ts_kernel<FMT, TsProj>, m[0], m[1], m[2], m[3], q, ea);
}

static bool launch_ts_pass(cudaStream_t st, const GemvArgs& a, const TsPlan& p, int* err, bool* fused) {
  switch (a.format) {
    case F_Q4_0: return launch_ts_fmt<F_Q4_0>(st, a, p, err, fused);
    case F_Q8_0: return launch_ts_fmt<F_Q8_0>(st, a, p, err, fused);
    case F_Q6_K: return launch_ts_fmt<F_Q6_K>(st, a, p, err, fused);
    case F_MXFP8: return launch_ts_fmt<F_MXFP8>(st, a, p, err, fused);
    case F_NVFP4: return launch_ts_fmt<F_NVFP4>(st, a, p, err, fused);
    default: return launch_ts_fmt<F_MXFP4>(st, a, p, err, fused);
  }
}

bool launch_ts(cudaStream_t st, const GemvArgs& a, bool* fused) {
  *fused = false;
  TsPlan p;
  if (!ts_preferred(a) || !ts_projection_plan(a, &p) || !a.scratch || a.scratch_bytes < p.scratch()) return false;
  int* err = device_error_flag();
  if (!err) return false;
  const int64_t per = (int64_t)p.mg * p.groups;
  for (int64_t m0 = 0; m0 < a.M; m0 += per) {
    GemvArgs b = a;
    b.M = a.M - m0 < per ? a.M - m0 : per;
    b.x = (const char*)a.x + (size_t)m0 * a.K * 2;
    b.y = (char*)a.y + (size_t)m0 * a.N * (a.out_f32 ? 4 : 2);
    if (a.residual) b.residual = (const char*)a.residual + (size_t)m0 * a.N * 2;
    if (a.q_codes && a.out_quant == OQ_MXFP8) b.q_codes = (char*)a.q_codes + (size_t)m0 * (a.N / 32) * 33;
    TsPlan pb = p;
    if (m0 + per > a.M && m0 > 0 && (!ts_projection_plan(b, &pb) || pb.scratch() > a.scratch_bytes)) return false;
    if (!launch_ts_pass(st, b, pb, err, fused)) return false;
  }
  return true;
}

}  // namespace qx
