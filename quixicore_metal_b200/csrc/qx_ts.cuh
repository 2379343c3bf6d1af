// Packed-weight contraction with the decoded weights as the TENSOR-MEMORY operand of tcgen05.mma.
//
//   out[n, m] = sum_k W[n, k] * x[m, k]        W packed (q4_0, q8_0, q6_K, mxfp8, nvfp4, mxfp4)
//
// The weight rows are the M-mode of the MMA (128 rows = 128 TMEM lanes), the activation rows its
// N-mode.  A worker thread owns one weight row: it reads the row's packed bytes from shared memory,
// decodes them in registers and writes them to its TMEM lane with tcgen05.st; the tensor core reads
// A from there.  Why not the usual shared-memory operand (measured, M = 128, K = 16, clocks per MMA):
//     N =            16    32    64   128
//     A in shared    39    40    48    64      (bound by reading A: 4 KB per MMA)
//     A in TMEM       9    16    32    64      (the full rate of the tensor core at every N)
// so a decode batch costs the tensor core what it must and no more, the operand needs no swizzled
// stores, no proxy fence and no shared-memory bandwidth, and one kernel serves 2 .. 256 rows.
// One thread chosen by elect.sync issues the MMAs: behind a `lane == 0` test each issue costs 112 clocks.
//
// Exactness.  All operands are f16 and every product term is exact:
//   * activations are row-scaled f16 (largest magnitude in [2^14, 2^15)), as everywhere on this path;
//   * nvfp4, mxfp4, mxfp8: weight x block scale (x a fixed power of two) has at most 6 significant bits;
//   * q4_0: w = (n - 8) * d is split as (n - 8) * dh + (n - 8) * dl, dh = the upper 7 bits of d, dl the
//     rest: both products fit 11 bits.  Two terms, two MMAs into the same accumulator;
//   * q8_0: hi = f16(q * d), lo = fma(q, d, -hi): q * d has 19 bits and is a multiple of 2^-24 (the
//     spacing of f16 subnormals, which the tensor core keeps), so lo is exact;
//   * q6_K: w = q * (sc * d), at most 24 bits, in three terms the same way.
// The accumulator is the fp32 dequantise-then-dot up to summation order.  The e8m0 formats hold 22 (mxfp8) and 28
// (mxfp4) exponents that way, around the exponent of ordinary weights; a row whose first block lies away from it
// (the rows of tokens that no training step has touched) is shifted by a power of two of its own, which the output
// warps take back (ts_row_shift).  Blocks whose scale still leaves the range - more than three decimal orders between the
// blocks of one row, or |d| >= 512, q6_K 16 - count as zeros and mark their row, and the output warps add their share
// to marked rows with fp32 arithmetic (ts_add_left_out).
//
// Accumulation.  The tensor core truncates the fp32 accumulator after every MMA; over the K / 16 * TERMS
// MMAs of a row that is a bias towards zero of about 3e-8 per MMA (q8_0, K = 8192, one accumulator: 1.9e-5).
// So a chunk of TsFmt::CHUNK stages is accumulated at a time, and the accumulator warps add the chunks to
// running sums in TMEM with rounded fp32 additions (the same case: 6e-7; nvfp4, mxfp4, mxfp8: 2e-7).
//
// Roles (32 warps): 16 workers; 4 accumulator warps, which sum the chunks and write a finished segment to
// global scratch (L2); 8 output warps, which turn it into outputs (or token selections) while the others
// already work on the next segment; two MMA issuers (one per row block of an item: issuing the four MMAs of
// a slot is a chain of 100 - 200 clocks); a loader of weight boxes and a loader of activations.
// A raw stage is 256 columns of 128 rows, fetched as P TMA boxes (P = 1 when rows are 16-byte aligned;
// otherwise the matrix is seen as N / P super-rows of P rows, whose pitch is a multiple of 16, and box
// p holds the rows p, p + P, ... of the tile - their common misalignment is resolved by the decoder).
// The four worker groups take one 64-column quarter each (q6_K: halves of alternate stages) and hand it
// over as one slot of the TMEM operand ring.
//
// Work split: the flat list of (item, stage) units is cut into equal contiguous ranges, one per CTA,
// whatever N is.  The CTA whose part of a cut item arrives last (a ticket, no waiting) adds the parts in CTA
// order and makes the outputs.
#pragma once

#include <type_traits>
#include <utility>

#include "qx_formats.cuh"
#include "qx_tc.cuh"

namespace qx {

constexpr int TS_WORKERS = 16;                   // worker warps: 4 groups x 4 lane quadrants
constexpr int TS_SUM_WARP = 16, TS_SUM = 4;      // accumulator warps, one per lane quadrant
constexpr int TS_OUT_WARP = 20, TS_OUT = 8;      // output warps
constexpr int TS_MMA_WARP = 28;                  // two MMA issuers, then the loaders
constexpr int TS_RAW_WARP = 30, TS_ACT_WARP = 31, TS_WARPS = 32;
constexpr int TS_MARK_RING = 16;                 // segments the workers can be ahead of the output warps: at most 8
constexpr int TS_KC = 256;                       // columns per raw stage
constexpr int TS_MAX_RAW = 8, TS_MAX_ACT = 8, TS_MAX_SLOTS = 16;

template <int FMT> struct TsFmt;
// BYTES: packed bytes of 256 columns; PITCH: row pitch in shared memory = box width, an odd multiple of 16
// (the 8 rows of one 16-byte access phase fall into different bank groups) with room for the
// misalignment of its rows; TERMS: f16 terms per weight; CHUNK: raw stages summed by the tensor core
// before the fp32 sum is taken over; the accumulator times ACC_SCALE is the dot.
template <> struct TsFmt<F_Q4_0>  { static constexpr int BK = 32,  BB = 18,  BYTES = 144, PITCH = 144, TERMS = 2, GPS = 4, CHUNK = 1; static constexpr float ACC_SCALE = 1.f; };
template <> struct TsFmt<F_Q8_0>  { static constexpr int BK = 32,  BB = 34,  BYTES = 272, PITCH = 272, TERMS = 2, GPS = 4, CHUNK = 1; static constexpr float ACC_SCALE = 1.f; };
template <> struct TsFmt<F_Q6_K>  { static constexpr int BK = 256, BB = 210, BYTES = 210, PITCH = 240, TERMS = 3, GPS = 2, CHUNK = 1; static constexpr float ACC_SCALE = 1.f; };
template <> struct TsFmt<F_MXFP8> { static constexpr int BK = 32,  BB = 33,  BYTES = 264, PITCH = 272, TERMS = 1, GPS = 4, CHUNK = 2; static constexpr float ACC_SCALE = 0x1p-9f; };
template <> struct TsFmt<F_NVFP4> { static constexpr int BK = 16,  BB = 9,   BYTES = 144, PITCH = 144, TERMS = 1, GPS = 4, CHUNK = 8; static constexpr float ACC_SCALE = 256.f; };
template <> struct TsFmt<F_MXFP4> { static constexpr int BK = 32,  BB = 17,  BYTES = 136, PITCH = 144, TERMS = 1, GPS = 4, CHUNK = 8; static constexpr float ACC_SCALE = 0x1p-12f; };

// Position of column c (0 <= c < 32) of a 32-column unit in the prepared activation row: the order in
// which the decoders below emit their f16 pairs.
__host__ __device__ inline int ts_position(int fmt, int c) {
  switch (fmt) {
    case F_Q4_0: { const int hi = c >> 4, r = c & 15, t = r >> 2, i = r & 3;      // words (4t,4t+2) (16+4t,..) (4t+1,4t+3) (16+4t+1,..)
                   return 2 * (4 * t + 2 * (i & 1) + hi) + (i >> 1); }
    case F_NVFP4: { const int r = c & 15; return (c & 16) | ((r & 7) << 1) | (r >> 3); }
    case F_MXFP4: return ((c & 15) << 1) | (c >> 4);
    default: return c;
  }
}

// ---- plan (host) and kernel parameters ---------------------------------------------------------------
struct TsPlan {
  int rb, dual;            // row blocks of 128 per item (dual: block 0 = gate rows, block 1 = up rows)
  int nb, mp, mg, groups;  // MMA N; rows per 16-byte column chunk of the activation image; rows per group; groups
  int P;                   // row interleave (see above)
  int tiles, tile_rows, nks, items;
  int sums, nd, na;        // TMEM: running sums kept (else: one chunk per segment), chunk buffers, operand slots
  int issuers;             // MMA issuing warps: 2 (one per row block) when each has operand slots of its own
  int nraw;                // raw stages
  int nact;                // activation stages of 256 columns
  int whole;               // items are not cut between CTAs (no partials)
  unsigned grid;
  size_t smem, off_act, off_aux, off_bar;
  size_t img_bytes, scale_bytes, count_bytes, part_bytes;   // scratch
  size_t scratch() const { return img_bytes + scale_bytes + count_bytes + part_bytes; }
};

struct TsParams {
  TsPlan p;
  const uint8_t* w[2];
  const void* x; int x_bf16;                     // raw activations (marked rows)
  const uint8_t* img; const float* rowscale;     // prepared activations
  float* part; unsigned* count;
  int M, K, N;
  int* err;
};

// Plan of one call (qx_ts.cu): rb = row blocks per item (1 or 2; 2 with `dual`), max_group = most activation
// rows of one group, aux = shared memory the epilogue policy needs, may_cut = partial accumulators allowed.
// False: the shape is not served.
bool ts_plan(TsPlan* p, int format, int64_t M, int64_t K, int64_t N, int rb, int dual, int max_group, size_t aux, bool may_cut);
bool ts_shape_ok(int format, int64_t K, int64_t N, const void* w0, const void* w1);
// Tensor maps of one weight matrix: [0] the residues whose last super-row exists, [1] the others.
bool ts_maps(const TsPlan& p, int format, const void* w, int64_t K, int64_t N, CUtensorMap* m);
// Prepared activations of a call into scratch (carved by the plan's byte counts); zeroes the tickets.  False: not
// launched, and the contraction must not be.
struct TsScratch { uint8_t* img; float* rowscale; unsigned* count; float* part; };
TsScratch ts_carve(const TsPlan& p, void* scratch);
bool ts_launch_prep(cudaStream_t st, const TsPlan& p, int format, const void* x, qx_dtype dtype, const TsScratch& s, int M, int K);

// A launch that may start before its predecessor in the stream has finished (the kernels here call
// griddepcontrol.wait before they touch what it produces; the contraction's weights are complete when it starts, see
// prep_rows_kernel).
template <typename... P, typename... A>
bool ts_launch_dependent(cudaStream_t st, dim3 grid, dim3 block, size_t smem, void (*kernel)(P...), A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...) == cudaSuccess) { note_launch(); return true; }
  cudaGetLastError();
  return false;
}

// What an output policy sees: one finished item as `parts` fp32 arrays [row block][column][128 rows] in global
// scratch (one array unless the item was cut), column = activation row of the group, row = weight row inside
// the block.  Columns m_count .. nb - 1 hold nothing of use.
struct TsItem {
  int tile, m_base, m_count;
  const float* first; const float* rest; size_t step; int parts;     // part 0, then rest + (k - 1) * step
  __device__ __forceinline__ const float* part(int k) const { return k == 0 ? first : rest + (size_t)(k - 1) * step; }
};

__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
  return r != 0;
}
// The MMAs of one operand slot (64 columns: four K = 16 steps, TERMS f16 terms each, 32 columns of TMEM apart)
// and the commit that frees it.  A whole warp calls it; the instructions are predicated on one elected lane
// inside the asm block, without a branch: behind an `if (elect)` in a loop the operands are moved to
// uniform registers anew for every instruction (four MMAs and a commit: 270 clocks against 60 here).
// `fresh` = 0: the first MMA starts the accumulator.
#define QX_TS_MMA(A, KK, PRED) \
  "add.u32 m, %1, " #A ";\n\tmad.lo.u32 l, %4, " #KK ", %2;\n\tmov.b64 b, {l, %3};\n\t" \
  "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [m], b, %5, " #PRED ";\n\t"
template <int TERMS>
__device__ __forceinline__ void ts_mma_slot(uint32_t d, uint32_t a, uint32_t blo, uint32_t bhi, uint32_t bk, uint32_t idesc,
                                            uint32_t fresh, uint32_t bar) {
#define QX_TS_HEAD "{\n\t.reg .pred e, p, t;\n\t.reg .b64 b;\n\t.reg .b32 l, m;\n\telect.sync _|e, 0xffffffff;\n\t" \
                   "setp.ne.b32 p, %6, 0;\n\tsetp.eq.u32 t, 0, 0;\n\t"
#define QX_TS_TAIL "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%7];\n\t}"
#define QX_TS_ARGS ::"r"(d), "r"(a), "r"(blo), "r"(bhi), "r"(bk), "r"(idesc), "r"(fresh), "r"(bar) : "memory"
  if constexpr (TERMS == 1)
    asm volatile(QX_TS_HEAD QX_TS_MMA(0, 0, p) QX_TS_MMA(8, 1, t) QX_TS_MMA(16, 2, t) QX_TS_MMA(24, 3, t) QX_TS_TAIL QX_TS_ARGS);
  else if constexpr (TERMS == 2)
    asm volatile(QX_TS_HEAD QX_TS_MMA(0, 0, p) QX_TS_MMA(32, 0, t) QX_TS_MMA(8, 1, t) QX_TS_MMA(40, 1, t) QX_TS_MMA(16, 2, t)
                 QX_TS_MMA(48, 2, t) QX_TS_MMA(24, 3, t) QX_TS_MMA(56, 3, t) QX_TS_TAIL QX_TS_ARGS);
  else
    asm volatile(QX_TS_HEAD QX_TS_MMA(0, 0, p) QX_TS_MMA(32, 0, t) QX_TS_MMA(64, 0, t) QX_TS_MMA(8, 1, t) QX_TS_MMA(40, 1, t)
                 QX_TS_MMA(72, 1, t) QX_TS_MMA(16, 2, t) QX_TS_MMA(48, 2, t) QX_TS_MMA(80, 2, t) QX_TS_MMA(24, 3, t)
                 QX_TS_MMA(56, 3, t) QX_TS_MMA(88, 3, t) QX_TS_TAIL QX_TS_ARGS);
}
__device__ __forceinline__ void ts_commit_elected(uint32_t bar) {
  asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
               "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
}
// Shared-memory operand without swizzle, K-major: 8-row x 16-byte core matrices, `lbo16` 16-byte units from
// one to the next along K, 128 bytes along N.  With fewer than 8 rows the core matrices overlap: row r of
// chunk c is read at c * lbo16 + r, which for r >= mp is another chunk's data - columns nobody reads.
__device__ __forceinline__ uint64_t umma_desc_plain(uint32_t addr, int lbo16) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)lbo16 << 16) | ((uint64_t)(128 >> 4) << 32) | ((uint64_t)1 << 46);
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds64v(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t h2fms(uint32_t a, uint32_t b, uint32_t c) {      // a * b - c
  const __half2 r = __hfma2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b),
                            __hneg2(*reinterpret_cast<const __half2*>(&c)));
  return *reinterpret_cast<const uint32_t*>(&r);
}

// ---- decoders: 64 columns (one quarter of a raw stage) of this thread's row ------------------------------
// load<J>(): the packed words of quarter J, moved so that w[0] starts with the quarter's first byte: the quarters
// have different alignments, and one copy of the decoding code for all of them (a moved word costs one
// instruction) keeps the kernel's hot code small - with a copy per quarter the issuers waited for
// instructions more than for anything else (q8_0, 64 rows: 118 us against 98).
// batch<S>(): columns 16 S .. 16 S + 15 -> 8 words per term; returns false when a block's scale is outside the
// exact range (its words are then finite placeholders).
template <int FMT> struct TsDec {
  using F = TsFmt<FMT>;
  static constexpr int LEN = (64 / F::BK) * F::BB;                 // bytes of a quarter
  static constexpr bool WIDE = F::BYTES % 16 == 0;                 // chunk 16-byte aligned: 16-byte loads, else 8
  static constexpr int UNIT = WIDE ? 16 : 8;
  static constexpr int NW = (LEN + 3) / 4;
  static constexpr int REL = 0;
  uint32_t w[NW];
  uint32_t base;                                                   // e8m0 formats: the block exponent that makes an f16 exponent of 0
  static constexpr uint32_t BASE = FMT == F_MXFP8 ? 95u : 100u;    // ... of a row that is not shifted

  template <int J> __device__ __forceinline__ void load(uint32_t addr) {
    constexpr int START = J * LEN, BASE = START / UNIT * UNIT, OFF = START - BASE;
    constexpr int NLD = (START + LEN + UNIT - 1) / UNIT - START / UNIT;
    uint32_t v[NLD * UNIT / 4 + 1];
    v[NLD * UNIT / 4] = 0u;
#pragma unroll
    for (int i = 0; i < NLD; ++i) {
      if constexpr (WIDE) {
        const uint4 t = lds128(addr + BASE + 16 * i);
        v[4 * i] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w;
      } else {
        const uint2 t = lds64v(addr + BASE + 8 * i);
        v[2 * i] = t.x; v[2 * i + 1] = t.y;
      }
    }
#pragma unroll
    for (int i = 0; i < NW; ++i)
      w[i] = OFF % 4 == 0 ? v[OFF / 4 + i] : __funnelshift_r(v[OFF / 4 + i], v[OFF / 4 + i + 1], (OFF % 4) * 8);
  }
  template <int B> __device__ __forceinline__ uint32_t get32() const {          // 32 bits at byte B of the loaded words
    if constexpr (B % 4 == 0) return w[B / 4];
    else return __funnelshift_r(w[B / 4], w[B / 4 + 1], (B % 4) * 8);
  }
  // byte B in both halves, at bits [15:8] and [31:24] (low bytes zero)
  template <int B> __device__ __forceinline__ uint32_t byte_high() const {
    return __byte_perm(w[B / 4], 0u, 0x0404 | (B % 4) << 4 | (B % 4) << 12);
  }
  template <int B> __device__ __forceinline__ uint32_t half_pair() const {      // the 16 bits at byte B in both halves
    if constexpr (B % 4 == 3) return __byte_perm(w[B / 4], w[B / 4 + 1], 0x4343);
    else return __byte_perm(w[B / 4], 0u, 0x1010 + 0x1111 * (B % 4));
  }
  template <int B> __device__ __forceinline__ uint32_t byte() const { return (w[B / 4] >> ((B % 4) * 8)) & 0xFFu; }

  template <int S> __device__ __forceinline__ bool batch(uint32_t (&hi)[8], uint32_t (&lo)[8]) const {
    if constexpr (FMT == F_NVFP4) {
      constexpr int B = REL + 9 * S;                               // one 16-column block
      const uint32_t v = byte_high<B>();
      const uint32_t s2 = e4m3_bits(v);                            // scale * 2^-8
      const uint32_t c[2] = {get32<B + 1>(), get32<B + 5>()};
#pragma unroll
      for (int i = 0; i < 2; ++i) e2m1_word(c[i], s2, hi + 4 * i);
      return true;
    } else {
      constexpr int BLK = REL + (S >> 1) * F::BB;                  // the 32-column block's first byte
      constexpr int HALF = S & 1;
      if constexpr (FMT == F_MXFP4) {
        const uint32_t e = byte<BLK>();
        const uint32_t c[2] = {get32<BLK + 1 + 8 * HALF>(), get32<BLK + 5 + 8 * HALF>()};
        // 2^(e - 127 + 12) as f16: exact products for 101 <= e <= 128 (less the shift of the row)
        uint32_t s2 = ((e - base) << 10) * 0x00010001u;
        bool ok = true;
        if (e - base - 1u > 27u) {
          ok = ((c[0] | c[1]) & 0x77777777u) == 0u;
          s2 = 0u;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) e2m1_word(c[i], s2, hi + 4 * i);
        return ok;
      } else if constexpr (FMT == F_MXFP8) {
        const uint32_t e = byte<BLK>();
        const uint32_t c[4] = {get32<BLK + 1 + 16 * HALF>(), get32<BLK + 5 + 16 * HALF>(), get32<BLK + 9 + 16 * HALF>(),
                               get32<BLK + 13 + 16 * HALF>()};
        // code bits moved under the f16 exponent are value * 2^-8 for every code (subnormals and 0x7F = 480, which
        // the hardware converter reads as NaN, included); times 2^(e - 127 + 17): exact for 104 <= e <= 125 (less the shift)
        uint32_t s2 = ((e - base) << 10) * 0x00010001u;
        bool ok = true;
        if (e - base - 9u > 21u) {
          ok = ((c[0] | c[1] | c[2] | c[3]) & 0x7F7F7F7Fu) == 0u;
          s2 = 0u;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          hi[2 * i] = h2mul(e4m3_bits(__byte_perm(c[i], 0u, 0x1404)), s2);
          hi[2 * i + 1] = h2mul(e4m3_bits(__byte_perm(c[i], 0u, 0x3424)), s2);
        }
        return ok;
      } else if constexpr (FMT == F_Q4_0) {
        uint32_t d2 = half_pair<BLK>();
        const bool ok = (d2 & 0x7C00u) < 0x6000u;                  // |d| < 512
        if (!ok) d2 = 0u;
        const uint32_t dh = d2 & 0xFFF0FFF0u, dl = h2sub(d2, dh);
        const uint32_t ah = h2mul(dh, 0x54005400u), ch = h2mul(dh, 0xD480D480u);   // 64 dh, -72 dh
        const uint32_t al = h2mul(dl, 0x54005400u), cl = h2mul(dl, 0xD480D480u);
        q4_word<BLK + 2 + 8 * HALF>(0, ah, ch, al, cl, hi, lo);
        q4_word<BLK + 6 + 8 * HALF>(4, ah, ch, al, cl, hi, lo);
        return ok;
      } else {
        static_assert(FMT == F_Q8_0, "format");
        uint32_t d2 = half_pair<BLK>();
        const bool ok = (d2 & 0x7C00u) < 0x6000u;
        if (!ok) d2 = 0u;
        q8_word<BLK + 2 + 16 * HALF>(0, d2, hi, lo);  q8_word<BLK + 6 + 16 * HALF>(2, d2, hi, lo);
        q8_word<BLK + 10 + 16 * HALF>(4, d2, hi, lo); q8_word<BLK + 14 + 16 * HALF>(6, d2, hi, lo);
        return ok;
      }
    }
  }
  __device__ __forceinline__ static void e2m1_word(uint32_t c, uint32_t s2, uint32_t* o) {
    o[0] = h2mul(cvt_e2m1x2<0>(c), s2); o[1] = h2mul(cvt_e2m1x2<1>(c), s2);
    o[2] = h2mul(cvt_e2m1x2<2>(c), s2); o[3] = h2mul(cvt_e2m1x2<3>(c), s2);
  }
  __device__ __forceinline__ static uint32_t e4m3_bits(uint32_t v) {            // codes at [15:8] and [31:24]
    return ((v >> 1) & 0x3F803F80u) | (v & 0x80008000u);
  }
  // A nibble moved to mantissa bits 4..7 under the exponent of 1 is 1 + n / 64; one fma per term makes
  // 64 d (1 + n / 64) - 72 d = (n - 8) d of it.
  template <int B> __device__ __forceinline__ void q4_word(int at, uint32_t ah, uint32_t ch, uint32_t al, uint32_t cl,
                                                           uint32_t (&hi)[8], uint32_t (&lo)[8]) const {
    const uint32_t v = get32<B>();
    const uint32_t m[4] = {((v << 4) & 0x00F000F0u) | 0x3C003C00u, (v & 0x00F000F0u) | 0x3C003C00u,
                           ((v >> 4) & 0x00F000F0u) | 0x3C003C00u, ((v >> 8) & 0x00F000F0u) | 0x3C003C00u};
#pragma unroll
    for (int i = 0; i < 4; ++i) { hi[at + i] = h2fma(m[i], ah, ch); lo[at + i] = h2fma(m[i], al, cl); }
  }
  template <int B> __device__ __forceinline__ void q8_word(int at, uint32_t d2, uint32_t (&hi)[8], uint32_t (&lo)[8]) const {
    const uint32_t u = get32<B>() ^ 0x80808080u;
    const uint32_t q0 = h2sub(__byte_perm(u, 0x64646464u, 0x4140), 0x64806480u);
    const uint32_t q1 = h2sub(__byte_perm(u, 0x64646464u, 0x4342), 0x64806480u);
    hi[at] = h2mul(q0, d2);     lo[at] = h2fms(q0, d2, hi[at]);
    hi[at + 1] = h2mul(q1, d2); lo[at + 1] = h2fms(q1, d2, hi[at + 1]);
  }
};

// q6_K: 128 columns (half C of a 256-column super-block).  Blocks are only 2-byte aligned: 8-byte loads,
// one select and one funnel shift per word bring the bytes into place.
struct TsDecQ6 {
  uint32_t q[16], h[8], sc[2], d;
  template <int N> __device__ __forceinline__ static void fetch(uint32_t addr, uint32_t (&o)[N]) {
    const uint32_t a8 = addr & ~7u;
    const bool up = (addr & 4u) != 0u;
    const uint32_t sh = (addr & 2u) * 8u;
    uint32_t v[2 * ((N + 3) / 2)];
#pragma unroll
    for (int i = 0; i < (N + 3) / 2; ++i) { const uint2 t = lds64v(a8 + 8 * i); v[2 * i] = t.x; v[2 * i + 1] = t.y; }
    uint32_t s[N + 1];
#pragma unroll
    for (int i = 0; i <= N; ++i) s[i] = up ? v[i + 1] : v[i];
#pragma unroll
    for (int i = 0; i < N; ++i) o[i] = __funnelshift_r(s[i], s[i + 1], sh);
  }
  __device__ __forceinline__ void load(uint32_t addr, int c) {
    fetch(addr + 64 * c, q);
    fetch(addr + 128 + 32 * c, h);
    fetch(addr + 192 + 8 * c, sc);
    d = lds16(addr + 208);
  }
  // columns 16 * SB .. 16 * SB + 15 of the half (SB = 0..7): one sub-block
  template <int SB> __device__ __forceinline__ void batch(uint32_t d2, uint32_t (&hi)[8], uint32_t (&mid)[8], uint32_t (&lo)[8]) const {
    constexpr int B = SB >> 1, T0 = (SB & 1) * 4;                  // 32-column quarter; first word of its 8 (ql, qh)
    const uint32_t s8 = __byte_perm(sc[SB >> 2] ^ 0x80808080u, 0x64646464u, 0x4040 + 0x0101 * (SB & 3));
    const uint32_t s2 = h2sub(s8, 0x64806480u);                    // the sub-scale, both halves
    const uint32_t th = h2mul(s2, d2), tl = h2fms(s2, d2, th);     // sc * d = th + tl
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const uint32_t Q = q[(B & 1) * 8 + T0 + t], H = h[T0 + t];
      const uint32_t q4 = B < 2 ? Q : (Q >> 4);
      const uint32_t h2 = B == 0 ? (H << 4) : (B == 1 ? (H << 2) : (B == 2 ? H : (H >> 2)));
      const uint32_t c = (q4 & 0x0F0F0F0Fu) | (h2 & 0x30303030u);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const uint32_t v = h2sub(__byte_perm(c, 0x64646464u, e ? 0x4342 : 0x4140), 0x64206420u);   // code - 32
        const uint32_t p1 = h2mul(v, th), p2 = h2fms(v, th, p1);
        const uint32_t r = h2fma(v, tl, p2);
        hi[2 * t + e] = p1; mid[2 * t + e] = r; lo[2 * t + e] = h2fma(v, tl, h2sub(p2, r));
      }
    }
  }
};

// slot row L of a raw stage -> row inside its 128-row block (P > 1: box r holds the rows r, r + P, ...)
__device__ __forceinline__ int ts_row_of(int P, int L) { return P == 1 ? L : (L % (128 / P)) * P + L / (128 / P); }

// ---- rows away from the ordinary exponents (e8m0 formats) ---------------------------------------------------
// A row's weights are decoded times 2^shift: 0 while the exponent e of its first block is that of ordinary weights
// (largest of a block 0.003 to 1.7, mxfp4 6e-6 to 0.7) or the block holds nothing, else what moves e to 114, the middle
// of the range; no further than TsDec::base stays positive and an exponent of 255 (infinity) out of every range.
template <int FMT> constexpr bool ts_shifts() { return FMT == F_MXFP8 || FMT == F_MXFP4; }
// Called by whole warps.
template <int FMT>
__device__ __forceinline__ int ts_row_shift(uint32_t e, const uint8_t* row) {
  const bool far = !(FMT == F_MXFP8 ? e - 110u <= 9u : e - 107u <= 17u) & (e != 255u);
  if (!__any_sync(0xffffffffu, far)) return 0;
  uint32_t any = 0u;
#pragma unroll 1
  for (int i = 1; i < TsFmt<FMT>::BB; i += 8) {                      // (rows that hold something show it in their first codes)
#pragma unroll
    for (int k = 0; k < 8; ++k) any |= __ldg(row + i + k) & (FMT == F_MXFP8 ? 0x7Fu : 0x77u);
    if (!__any_sync(0xffffffffu, far & (any == 0u))) break;
  }
  const int shift = min(max(114 - (int)e, (FMT == F_MXFP8 ? 125 : 128) - 254), 95);
  return far & (any != 0u) ? shift : 0;
}
__device__ __forceinline__ float ts_pow2(int n) { return __uint_as_float(n < -126 ? 0x00400000u : (uint32_t)(n + 127) << 23); }   // -127 <= n

// ---- blocks outside the exact range ------------------------------------------------------------------------
// The decoders put zeros in their place and mark the row; their share of the dot is added to the finished segment.
// Whether 32-column block b of a row is one of them (shift: ts_row_shift of the row).
template <int FMT>
__device__ __forceinline__ bool ts_block_left_out(const uint8_t* row, int b, int shift) {
  if constexpr (FMT == F_Q6_K) {
    const uint8_t* d = row + (size_t)(b >> 3) * 210 + 208;
    return (__ldg(d + 1) & 0x7Cu) >= 0x4Cu;
  } else if constexpr (FMT == F_Q4_0 || FMT == F_Q8_0) {
    return (__ldg(row + (size_t)b * TsFmt<FMT>::BB + 1) & 0x7Cu) >= 0x60u;
  } else {
    const uint8_t* blk = row + (size_t)b * TsFmt<FMT>::BB;
    const uint32_t x = __ldg(blk) - (TsDec<FMT>::BASE - (uint32_t)shift);
    uint32_t any = 0u;
#pragma unroll 1
    for (int i = 1; i < TsFmt<FMT>::BB; ++i) any |= __ldg(blk + i);
    return !(FMT == F_MXFP8 ? x - 9u <= 21u : x - 1u <= 27u) & ((any & (FMT == F_MXFP8 ? 0x7Fu : 0x77u)) != 0u);
  }
}
// weight i of 32-column block b
template <int FMT>
__device__ __forceinline__ float ts_weight(const uint8_t* row, int b, int i) {
  if constexpr (FMT == F_Q6_K) {
    const uint8_t* s = row + (size_t)(b >> 3) * 210;
    const int half = (b >> 2) & 1, g = b & 3;
    const uint32_t l = (uint32_t)__ldg(s + 64 * half + 32 * (g & 1) + i) >> (4 * (g >> 1)), h = (uint32_t)__ldg(s + 128 + 32 * half + i) >> (2 * g);
    const float d = f16_bits_to_f32(__ldg(s + 208), __ldg(s + 209)) * (float)(int)(int8_t)__ldg(s + 192 + 8 * half + 2 * g + (i >> 4));
    return d * (float)((int)((l & 15u) | (h & 3u) << 4) - 32);
  } else {
    const uint8_t* s = row + (size_t)b * TsFmt<FMT>::BB;
    if constexpr (FMT == F_Q8_0) return f16_bits_to_f32(__ldg(s), __ldg(s + 1)) * (float)(int)(int8_t)__ldg(s + 2 + i);
    else if constexpr (FMT == F_MXFP8) return e8m0_to_f32(__ldg(s)) * e4m3_to_f32(__ldg(s + 1 + i));
    else {
      const uint32_t n = ((uint32_t)__ldg(s + (FMT == F_Q4_0 ? 2 : 1) + (i & 15)) >> (4 * (i >> 4))) & 15u;
      return FMT == F_Q4_0 ? f16_bits_to_f32(__ldg(s), __ldg(s + 1)) * (float)((int)n - 8) : e8m0_to_f32(__ldg(s)) * e2m1_to_f32(n);
    }
  }
}
// The marked rows of a quadrant (mk: 4 words from one row block to the next) of a segment, over its stored accumulators
// (`out`: [row block][column][128 rows]), by one warp; a lane takes a column.  Rolled and inline: a call here costs every
// launch registers (64-row LM heads 5 %).
// 64 rows, mxfp8, 4096 -> 14336, 31.4 us: one block left out of one row 36.5, of 32 and 256 rows all over the matrix 39.6 and
// 40.7.  Making whole rows again in fp32 took 244 us for one and 4.2 ms for 32 of them.
template <int FMT>
__device__ __forceinline__ void ts_add_left_out(const TsParams& q, float* out, const uint32_t* mk, int quad, int tile, int m_base, int m_count,
                                                int ks0, int ks1, int lane) {
  const TsPlan& p = q.p;
#pragma unroll 1
  for (int rb = 0; rb < p.rb; ++rb)
#pragma unroll 1
    for (uint32_t bits = __reduce_or_sync(0xffffffffu, mk[rb * 4]); bits; bits &= bits - 1u) {
      const int row = ts_row_of(p.P, quad * 32 + __ffs(bits) - 1), n = tile * p.tile_rows + (p.dual ? 0 : rb * 128) + row;
      if (n >= q.N) continue;
      const uint8_t* w = q.w[p.dual ? rb : 0] + (size_t)n * ((size_t)(q.K / TsFmt<FMT>::BK) * TsFmt<FMT>::BB);
      int shift = 0;
      if constexpr (ts_shifts<FMT>()) shift = ts_row_shift<FMT>(__ldg(w), w);
      const float unit = ts_shifts<FMT>() ? TsFmt<FMT>::ACC_SCALE * ts_pow2(-shift) : TsFmt<FMT>::ACC_SCALE;
#pragma unroll 1
      for (int b0 = ks0 * 8; b0 < ks1 * 8; b0 += 32) {
        const int bl = min(b0 + lane, ks1 * 8 - 1);
        uint32_t left = __ballot_sync(0xffffffffu, ts_block_left_out<FMT>(w, bl, shift) & (b0 + lane < ks1 * 8));
#pragma unroll 1
        for (; left; left &= left - 1u) {
          const int b = b0 + __ffs(left) - 1;
#pragma unroll 1
          for (int c0 = 0; c0 < m_count; c0 += 32) {
            const int c = min(c0 + lane, m_count - 1);
            const uint16_t* x = reinterpret_cast<const uint16_t*>(q.x) + (size_t)(m_base + c) * q.K + b * 32;
            float a = 0.f;
#pragma unroll 1
            for (int i = 0; i < 32; ++i)
              a = fmaf(q.x_bf16 ? __uint_as_float((uint32_t)__ldg(x + i) << 16) : __half2float(__ushort_as_half(__ldg(x + i))),
                       ts_weight<FMT>(w, b, i), a);
            float* o = out + ((size_t)rb * p.nb + c) * 128 + row;
            const float v = __ldcg(o) + a / (q.rowscale[m_base + c] * unit);
            if (c0 + lane < m_count) __stcg(o, v);
          }
        }
      }
    }
}

// Marks the rows of a warp (bit = lane) that are not `ok`.  Without a branch, see ts_kernel.
__device__ __forceinline__ void ts_mark(uint32_t* word, bool ok, int lane) {
  const uint32_t bad = __ballot_sync(0xffffffffu, !ok);
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p red.shared.or.b32 [%0], %1;\n\t}" ::"r"(smem_u32(word)), "r"(bad),
               "r"(lane == 0 ? bad : 0u) : "memory");
}

// Position in a ring of n slots: index and phase parity.
struct TsRing {
  int slot; uint32_t par;
  __device__ __forceinline__ void advance1(int n) { if (++slot == n) { slot = 0; par ^= 1u; } }
  __device__ __forceinline__ void advance(int by, int n) { slot += by; par ^= (uint32_t)(slot / n) & 1u; slot %= n; }
};

// Unit ranges.  Activation groups run side by side: CTA b works on group b % groups, and the CTAs of a group
// cut its tiles * nks units evenly (CTAs of different groups walk the same tiles at the same time and
// share them through L2).
struct TsRange { int grp, cta, ctas, u0, u1; };      // the plan keeps tiles * nks below 2^30
__host__ __device__ inline TsRange ts_range(const TsPlan& p, int b) {
  TsRange r;
  r.grp = b % p.groups; r.cta = b / p.groups; r.ctas = (int)(p.grid / p.groups);
  const long long total = p.whole ? p.tiles : (long long)p.tiles * p.nks;
  r.u0 = (int)(total * r.cta / r.ctas); r.u1 = (int)(total * (r.cta + 1) / r.ctas);
  if (p.whole) { r.u0 *= p.nks; r.u1 *= p.nks; }
  return r;
}
// CTA (inside its group) that holds unit u
__device__ __forceinline__ int ts_owner(const TsPlan& p, int ctas, long long u) {
  return (int)(((u + 1) * ctas - 1) / ((long long)p.tiles * p.nks));
}

// Epi: struct Args; packs_rows(args): writes MXFP8 rows, which a later call may take as its weights;
//      run<SHIFT>(args, params, item, scale, back, aux, warp, warps, lane), called by `warps` warps together (8 or 24): the
//        dot product of column c is the sum of the parts times scale[c], with SHIFT also times back[128 * block + row];
//        `aux`: AUX bytes of shared memory of this warp's own;
//      tail(...) by the output warps after the last item.
// Code that a launch runs once or twice is kept rolled: it is fetched cold, at about 70 clocks per 8
// instructions (an epilogue unrolled over 16 columns took 12,000 clocks for its first item).
template <int FMT, class Epi>
__global__ void __launch_bounds__(TS_WARPS * 32, 1)
ts_kernel(const __grid_constant__ CUtensorMap map_a0, const __grid_constant__ CUtensorMap map_b0,
          const __grid_constant__ CUtensorMap map_a1, const __grid_constant__ CUtensorMap map_b1,
          const __grid_constant__ TsParams q, const typename Epi::Args ea) {
  using F = TsFmt<FMT>;
  constexpr int TERMS = F::TERMS, SLOT_COLS = 32 * TERMS, STAGE = 128 * F::PITCH, GPS = F::GPS;
  const TsPlan& p = q.p;
  extern __shared__ uint8_t ts_smem[];
  // a programmatic dependent may be scheduled; it waits for this grid's end, but not with its weight loads
  if (!Epi::packs_rows(ea)) asm volatile("griddepcontrol.launch_dependents;");
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)ts_smem + 127) & ~(uintptr_t)127);
  const uint32_t sbase = smem_u32(smem);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;

  const uint32_t bars = sbase + (uint32_t)p.off_bar;
  auto RAW_FULL = [&](int i) { return bars + 8u * (uint32_t)i; };
  auto RAW_EMPTY = [&](int i) { return bars + 8u * (uint32_t)(TS_MAX_RAW + i); };
  auto ACT_FULL = [&](int i) { return bars + 8u * (uint32_t)(2 * TS_MAX_RAW + i); };
  auto ACT_EMPTY = [&](int i) { return bars + 8u * (uint32_t)(2 * TS_MAX_RAW + TS_MAX_ACT + i); };
  constexpr int B3 = 2 * TS_MAX_RAW + 2 * TS_MAX_ACT;
  auto OP_FULL = [&](int i) { return bars + 8u * (uint32_t)(B3 + i); };
  auto OP_EMPTY = [&](int i) { return bars + 8u * (uint32_t)(B3 + TS_MAX_SLOTS + i); };
  constexpr int B4 = B3 + 2 * TS_MAX_SLOTS;
  auto ACC_FULL = [&](int buf, int rb) { return bars + 8u * (uint32_t)(B4 + buf * 2 + rb); };
  auto ACC_EMPTY = [&](int buf, int rb) { return bars + 8u * (uint32_t)(B4 + 4 + buf * 2 + rb); };
  auto SEG_FULL = [&](int i) { return bars + 8u * (uint32_t)(B4 + 8 + i); };
  auto SEG_EMPTY = [&](int i) { return bars + 8u * (uint32_t)(B4 + 10 + i); };
  constexpr int NB = B4 + 12;
  uint32_t* words = reinterpret_cast<uint32_t*>(smem + p.off_bar + 8 * NB);
  volatile uint32_t* tmem_slot = words;
  volatile uint32_t* ticket = words + 1;
  uint32_t* marks = words + 4;                      // [segment ring][2 row blocks][4 quadrants] marked rows
  float* scale = reinterpret_cast<float*>(words + 4 + TS_MARK_RING * 8);   // per activation row of the group
  float* back = scale + 128;                        // e8m0 formats: 2^-shift of the item's weight rows

  {
    for (int i = tid; i < NB; i += TS_WARPS * 32) {
      uint32_t n = 1;                                                 // full barriers of copies and commits
      if (i >= TS_MAX_RAW && i < 2 * TS_MAX_RAW) n = GPS * 4;         // RAW_EMPTY: the reading worker warps
      else if (i >= B3 && i < B3 + TS_MAX_SLOTS) n = 4;               // OP_FULL: the warps of a worker group
      else if (i >= B4 + 10) n = TS_OUT;                              // SEG_EMPTY
      else if (i >= B4 + 4) n = TS_SUM;                               // ACC_EMPTY, SEG_FULL
      else if (i >= 2 * TS_MAX_RAW + TS_MAX_ACT && i < B3) n = (uint32_t)p.issuers;   // ACT_EMPTY
      mbar_init(bars + 8u * (uint32_t)i, n);
    }
    for (int i = tid; i < TS_MARK_RING * 8; i += TS_WARPS * 32) marks[i] = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == TS_MMA_WARP) tmem_alloc(smem_u32((const void*)tmem_slot), 512u);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (tid == 0 && *tmem_slot != 0u) atomicExch(q.err, 6);             // the allocation is the whole of TMEM: base 0
  const int acc_cols = p.rb * p.nb;                                   // columns of one accumulator buffer
  const uint32_t acc_base = p.sums ? (uint32_t)acc_cols : 0u;         // running sums, chunk buffers, operand slots
  const uint32_t op_base = acc_base + (uint32_t)(p.nd * acc_cols);
  const int chunk = p.sums ? F::CHUNK : 0x40000000;                   // stages per chunk

  // Bounded wait of a whole warp.  The common case - the phase is complete - is one try and one uniform
  // branch (a vote): the roles are serial chains of single warps whose length bounds the pipeline, and a
  // divergent loop here costs 120 clocks.  After one expiry the warp stops waiting (and the flag is up).
  bool dead = false;
  auto wait = [&](uint32_t bar, uint32_t parity) -> bool {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    for (int n = dead ? 1 : (1 << 22); n > 0; --n)
      if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    if (!dead) { dead = true; atomicExch(q.err, 5); }
    return false;
  };

  const TsRange rg = ts_range(p, (int)blockIdx.x);
  const int nks = p.nks, rbn = p.rb;
  // A segment: the part of one item this CTA computes, stages [ks0, ks1) of `tile`
  auto segment = [&](int& u, int& tile, int& ks0, int& ks1) {
    tile = u / nks;
    ks0 = u - tile * nks;
    ks1 = min(nks, ks0 + (rg.u1 - u));
    u += ks1 - ks0;
  };
  const int seg_rows = 128 / p.P;
  // first byte of this CTA's weight row n of row block rb (rows past the matrix: the last one)
  auto row_start = [&](int rb, int n) {
    const size_t row_bytes = (size_t)(q.K / F::BK) * F::BB;
    return q.w[p.dual ? rb : 0] + (size_t)min(n + (p.dual ? 0 : rb * 128), q.N - 1) * row_bytes;
  };

  if (warp < TS_WORKERS) {
    // ============================ workers ============================
    const int quad = warp & 3, grp = warp >> 2;
    const int L = quad * 32 + lane;                                   // TMEM lane = slot row of the raw stage
    const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
    const uint32_t res_off = (uint32_t)((long long)(L / seg_rows) * ((long long)(q.K / F::BK) * F::BB) & 15);
    const uint32_t slot_at0 = sbase + (uint32_t)(L * F::PITCH);       // this row's slot in raw stage 0
    const uint32_t op_at0 = op_base + lane_sel + (uint32_t)(grp * SLOT_COLS);
    TsRing raw{0, 0};
    int opb = 0; uint32_t opar = 1u;                                  // first operand slot of the stage, parity of its "empty"
    int stage_no = 0, nseg = 0;
    // e8m0 formats: TsDec::base of this thread's rows (low half: row block 0), made of the exponents of their first
    // blocks: from the raw stage that holds them, or from memory where the CTA starts inside an item
    uint32_t bases = 0u;
    const int wrow = ts_row_of(p.P, L);
    auto set_base = [&](int tile, int rb, uint32_t e) {
      const uint32_t b = TsDec<FMT>::BASE - (uint32_t)ts_row_shift<FMT>(e, row_start(rb, tile * p.tile_rows + wrow));
      bases = rb ? (bases & 0xFFFFu) | b << 16 : (bases & 0xFFFF0000u) | b;
    };
    if constexpr (ts_shifts<FMT>())
      if (rg.u0 < rg.u1 && rg.u0 % nks != 0)
        for (int rb = 0; rb < rbn; ++rb) set_base(rg.u0 / nks, rb, __ldg(row_start(rb, rg.u0 / nks * p.tile_rows + wrow)));
    for (int u = rg.u0; u < rg.u1; ++nseg) {
      int tile, ks0, ks1;
      segment(u, tile, ks0, ks1);
      uint32_t* mk = marks + (nseg & (TS_MARK_RING - 1)) * 8 + quad;
      if constexpr (FMT == F_Q6_K) {
        for (int ks = ks0; ks < ks1; ++ks) {
          const uint32_t off = (res_off + (uint32_t)(ks * F::BYTES)) & 15u;
          for (int rb = 0; rb < rbn; ++rb, ++stage_no, raw.advance1(p.nraw)) {
            if ((grp >> 1) != (stage_no & 1)) continue;
            wait(RAW_FULL(raw.slot), raw.par);
            TsDecQ6 dec;
            dec.load(slot_at0 + (uint32_t)(raw.slot * STAGE) + off, grp & 1);
            __syncwarp();
            if (lane == 0) mbar_arrive(RAW_EMPTY(raw.slot));
            const bool okrow = (dec.d & 0x7C00u) < 0x4C00u;           // |d| < 16
            const uint32_t d2 = okrow ? dec.d * 0x00010001u : 0u;
            ts_mark(mk + rb * 4, okrow, lane);
            uint32_t hi[8], mid[8], lo[8];
            auto put = [&](int s) {
              tmem_st8(op_at0 + 8 * s, hi); tmem_st8(op_at0 + 32 + 8 * s, mid); tmem_st8(op_at0 + 64 + 8 * s, lo);
            };
            auto open = [&](uint32_t parity) { wait(OP_EMPTY(grp), parity); __syncwarp(); tc_fence_after(); };
            auto done = [&]() {
              tmem_wait_st();
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(OP_FULL(grp));
            };
            // one operand slot per worker group, used for its two quarters in turn: even uses are first
            // quarters, odd ones second quarters
            dec.batch<0>(d2, hi, mid, lo); open(1u); put(0);
            dec.batch<1>(d2, hi, mid, lo); put(1);
            dec.batch<2>(d2, hi, mid, lo); put(2);
            dec.batch<3>(d2, hi, mid, lo); put(3); done();
            dec.batch<4>(d2, hi, mid, lo); open(0u); put(0);
            dec.batch<5>(d2, hi, mid, lo); put(1);
            dec.batch<6>(d2, hi, mid, lo); put(2);
            dec.batch<7>(d2, hi, mid, lo); put(3); done();
          }
        }
      } else {
        for (int ks = ks0; ks < ks1; ++ks) {
          const uint32_t off = F::BYTES % 16 == 0 ? 0u : (res_off + (uint32_t)(ks * F::BYTES)) & 15u;
          for (int rb = 0; rb < rbn; ++rb) {
            wait(RAW_FULL(raw.slot), raw.par);
            TsDec<FMT> dec;
            const uint32_t at = slot_at0 + (uint32_t)(raw.slot * STAGE) + off;
            if constexpr (ts_shifts<FMT>()) {
              if (ks == 0) set_base(tile, rb, lds8(at));
              dec.base = (bases >> (16 * rb)) & 0xFFFFu;
            }
            if (grp == 0) dec.template load<0>(at);
            else if (grp == 1) dec.template load<1>(at);
            else if (grp == 2) dec.template load<2>(at);
            else dec.template load<3>(at);
            __syncwarp();
            if (lane == 0) mbar_arrive(RAW_EMPTY(raw.slot));
            raw.advance1(p.nraw);
            const uint32_t dst = op_at0 + (uint32_t)(opb * SLOT_COLS);
            uint32_t hi[8], lo[8];
            auto put = [&](int s) {
              tmem_st8(dst + 8 * s, hi);
              if constexpr (TERMS == 2) tmem_st8(dst + 32 + 8 * s, lo);
            };
            bool okrow = dec.template batch<0>(hi, lo);
            wait(OP_EMPTY(opb + grp), opar);
            __syncwarp();
            tc_fence_after();
            put(0);
            okrow = dec.template batch<1>(hi, lo) && okrow; put(1);
            okrow = dec.template batch<2>(hi, lo) && okrow; put(2);
            okrow = dec.template batch<3>(hi, lo) && okrow; put(3);
            if constexpr (FMT != F_NVFP4) ts_mark(mk + rb * 4, okrow, lane);   // (whose scales are never out of range)
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(OP_FULL(opb + grp));
            opb += 4;
            if (opb == p.na) { opb = 0; opar ^= 1u; }
          }
        }
      }
    }
  } else if (warp < TS_OUT_WARP) {
    // ============================ accumulators ============================
    asm volatile("griddepcontrol.wait;" ::: "memory");                // the scratch may still be read by the kernel before
    const int quad = warp & 3;
    const int row = ts_row_of(p.P, quad * 32 + lane);
    const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
    const int m_count = min(p.mg, q.M - rg.grp * p.mg);
    TsRing acc{0, 0};
    int nseg = 0;
    for (int u = rg.u0; u < rg.u1; ++nseg) {
      int tile, ks0, ks1;
      segment(u, tile, ks0, ks1);
      const int nch = (ks1 - ks0 - 1) / chunk + 1;
      const bool summed = nch > 1;
      int last_buf = 0;
      for (int c = 0; c < nch; ++c) {
        const int buf = last_buf = acc.slot;
        for (int rb = 0; rb < rbn; ++rb) {
          wait(ACC_FULL(buf, rb), acc.par);
          __syncwarp();
          tc_fence_after();
          if (!summed) continue;
          const uint32_t src = acc_base + lane_sel + (uint32_t)(buf * acc_cols + rb * p.nb), dst = lane_sel + (uint32_t)(rb * p.nb);
#pragma unroll 1
          for (int c0 = 0; c0 < p.nb; c0 += 16) {
            uint32_t a[16];
            tmem_ld16_nowait(src + c0, a);
            if (c > 0) {
              uint32_t b[16];
              tmem_ld16_nowait(dst + c0, b);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 16; ++i) a[i] = __float_as_uint(__uint_as_float(a[i]) + __uint_as_float(b[i]));
            } else {
              tmem_wait_ld();
            }
            tmem_st16(dst + c0, a);
          }
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(ACC_EMPTY(buf, rb));
        }
        acc.advance1(p.nd);
      }
      const uint32_t acc_at = lane_sel + (summed ? 0u : acc_base + (uint32_t)(last_buf * acc_cols));
      // the finished segment -> scratch: slots 0 / 1 of the CTA for the head / tail part of a cut item, else 2 / 3 in turn
      const int sb = nseg & 1;
      wait(SEG_EMPTY(sb), ((uint32_t)(nseg >> 1) & 1u) ^ 1u);
      __syncwarp();
      const int kind = ks0 > 0 ? 0 : (ks1 < nks ? 1 : 2 + sb);
      float* out = q.part + ((size_t)(blockIdx.x * 4 + kind) * rbn) * p.nb * 128;
      for (int rb = 0; rb < rbn; ++rb)
#pragma unroll 1
        for (int c = 0; c < m_count; c += 8) {
          uint32_t r[8];
          tmem_ld8_nowait(acc_at + (uint32_t)(rb * p.nb + c), r);
          tmem_wait_ld();
          float* o = out + ((size_t)rb * p.nb + c) * 128 + row;
#pragma unroll
          for (int i = 0; i < 8; ++i) __stcg(o + i * 128, __uint_as_float(r[i]));
        }
      if (!summed) tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(SEG_FULL(sb));
        if (!summed)
          for (int rb = 0; rb < rbn; ++rb) mbar_arrive(ACC_EMPTY(last_buf, rb));
      }
    }
  } else if (warp < TS_MMA_WARP) {
    // outputs: below
  } else if (warp < TS_RAW_WARP) {
    // ============================ MMA issuers ============================
    const int rb0 = warp - TS_MMA_WARP, iss = p.issuers;
    if (rb0 < iss) {
      const uint32_t idesc = umma_idesc_f16(p.nb);
      const uint64_t bdesc0 = umma_desc_plain(sbase + (uint32_t)p.off_act, p.mp);
      const uint32_t bhi = (uint32_t)(bdesc0 >> 32), blo0 = (uint32_t)bdesc0;
      const uint32_t bk = 2u * (uint32_t)p.mp;                        // descriptor step of 16 columns
      int opb = 4 * rb0;                                              // first operand slot of this warp's next stage
      uint32_t opar = 0u;
      TsRing act{0, 0}, acc{0, 1};                                    // acc: chunk buffer and the parity of its "empty"
      int stage_no = 0;                                               // q6_K (one issuer)
      for (int u = rg.u0; u < rg.u1;) {
        int tile, ks0, ks1;
        segment(u, tile, ks0, ks1);
        int left = 0;                                                 // stages left in the chunk
        for (int ks = ks0; ks < ks1; ++ks) {
          const bool opens = left == 0;
          if (opens) left = chunk;
          --left;
          const bool closes = left == 0 || ks + 1 == ks1;
          const uint32_t bstage = blo0 + (uint32_t)act.slot * 16u * bk;  // 256 columns = 16 descriptor steps
          wait(ACT_FULL(act.slot), act.par);
          for (int rb = rb0; rb < rbn; rb += iss, ++stage_no) {
            const uint32_t d = acc_base + (uint32_t)(acc.slot * acc_cols + rb * p.nb);
            uint32_t fresh = opens ? 0u : 1u;                         // 0: the next MMA starts the accumulator
            if (opens) wait(ACC_EMPTY(acc.slot, rb), acc.par);
            // One warp's chain of steps bounds the pipeline up to 64 rows: everything that a slot needs advances by a constant.
            const int slot0 = FMT == F_Q6_K ? 2 * (stage_no & 1) : opb;
            uint32_t bar = OP_FULL(slot0), a = op_base + (uint32_t)(slot0 * SLOT_COLS), blo = bstage;
#pragma unroll 1
            for (int j = 0; j < 4; ++j, blo += 4 * bk) {
              wait(bar, FMT == F_Q6_K ? (uint32_t)(j & 1) : opar);
              tc_fence_after();
              ts_mma_slot<TERMS>(d, a, blo, bhi, bk, idesc, fresh, bar + 8u * TS_MAX_SLOTS);
              fresh = 1u;
              if (FMT != F_Q6_K || (j & 1)) { bar += 8u; a += SLOT_COLS; }
            }
            if (iss == 2 || rb == rbn - 1) ts_commit_elected(ACT_EMPTY(act.slot));
            if (closes) ts_commit_elected(ACC_FULL(acc.slot, rb));
            opb += 4 * iss;
            if (opb >= p.na) { opb -= p.na; opar ^= 1u; }
          }
          if (closes) { left = 0; acc.advance1(p.nd); }
          act.advance1(p.nact);
        }
      }
    }
  } else if (warp == TS_RAW_WARP) {
    // ============================ raw weight boxes ============================
    const int tail_res = q.N % p.P;                                   // residues whose last super-row exists: map a
    const long long row_bytes = (long long)(q.K / F::BK) * F::BB;
    TsRing raw{0, 0};
    int issued = 0;
    for (int u = rg.u0; u < rg.u1 && !dead;) {
      int tile, ks0, ks1;
      segment(u, tile, ks0, ks1);
      for (int ks = ks0; ks < ks1 && !dead; ++ks)
        for (int rb = 0; rb < rbn; ++rb) {
          if (!wait(RAW_EMPTY(raw.slot), raw.par ^ 1u)) break;
          const int row0 = tile * p.tile_rows + (p.dual ? 0 : rb * 128);
          const CUtensorMap* ma = p.dual && rb ? &map_a1 : &map_a0;
          const CUtensorMap* mb = p.dual && rb ? &map_b1 : &map_b0;
          const uint32_t dst = sbase + (uint32_t)(raw.slot * STAGE);
          if (elect_one()) {
            mbar_arrive_expect_tx(RAW_FULL(raw.slot), (uint32_t)STAGE);
            if (p.P == 1) {
              tma_box_2d(dst, ma, ((ks * F::BYTES) & ~15) >> 2, row0, RAW_FULL(raw.slot));
            } else {
              for (int r = 0; r < p.P; ++r) {
                const long long byte = r * row_bytes + (long long)ks * F::BYTES;
                tma_box_2d(dst + (uint32_t)(r * seg_rows * F::PITCH), r < tail_res ? ma : mb, (int)((byte & ~15ll) >> 1), row0 / p.P,
                           RAW_FULL(raw.slot));
              }
            }
          }
          __syncwarp();
          raw.advance1(p.nraw);
          ++issued;
        }
    }
    if (dead) {                                                       // boxes in flight must land before the CTA exits
      TsRing r{0, 0};
      r.advance(max(0, issued - p.nraw), p.nraw);
      for (int i = max(0, issued - p.nraw); i < issued; ++i, r.advance1(p.nraw))
        for (int k = 0; k < (1 << 20); ++k)
          if (mbar_try_wait(RAW_FULL(r.slot), r.par)) break;
    }
  } else {
    // ============================ activation stages ============================
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t bytes = (uint32_t)(TS_KC * p.mp * 2);
    const uint8_t* src = q.img + (size_t)rg.grp * q.K * p.mp * 2;
    TsRing act{0, 0};
    int issued = 0;
    const int depth = p.nact;
    for (int u = rg.u0; u < rg.u1 && !dead;) {
      int tile, ks0, ks1;
      segment(u, tile, ks0, ks1);
      for (int a = ks0; a < ks1; ++a) {
        if (!wait(ACT_EMPTY(act.slot), act.par ^ 1u)) break;
        if (elect_one()) {
          mbar_arrive_expect_tx(ACT_FULL(act.slot), bytes);
          bulk_g2s(sbase + (uint32_t)p.off_act + (uint32_t)act.slot * bytes, src + (size_t)a * bytes, bytes, ACT_FULL(act.slot));
        }
        __syncwarp();
        act.advance1(depth);
        ++issued;
      }
    }
    if (dead) {
      TsRing r{0, 0};
      r.advance(max(0, issued - depth), depth);
      for (int i = max(0, issued - depth); i < issued; ++i, r.advance1(depth))
        for (int k = 0; k < (1 << 20); ++k)
          if (mbar_try_wait(ACT_FULL(r.slot), r.par)) break;
    }
  }
  __syncwarp();

  if ((Epi::HELP && warp < TS_WORKERS) || (warp >= TS_OUT_WARP && warp < TS_MMA_WARP)) {
    // ============================ outputs ============================
    // Eight warps turn a segment into outputs while the others work on the next one.  With HELP the workers, which are done
    // when the last segment is, take their share of it, as it runs with nothing beside it (mxfp4, 256 rows, 8192 -> 28672,
    // MXFP8 rows out: 112,000 of 343,000 clocks).
    // It stands behind the roles, and its loops (as all of this kernel's) run on values that are the same for the whole warp
    // and that the compiler can see to be so - votes and reductions, not what a lane has loaded.  With a loop of each lane's
    // own count anywhere, or this code among the roles, all roles get by without uniform registers and with a reconvergence
    // point at every branch, and their chains set the pace (q8_0 and mxfp8, 200 rows, 4096 -> 14336: 103 and 97 us against
    // 71 and 76; nvfp4, 32 rows: 30 against 21).
    const bool helper = warp < TS_WORKERS;
    asm volatile("griddepcontrol.wait;" ::: "memory");                // all below reads or writes what the kernel before may
    const int ow = helper ? TS_OUT + warp : warp - TS_OUT_WARP, ot = ow * 32 + lane;
    const int m_base = rg.grp * p.mg, m_count = min(p.mg, q.M - m_base);
    uint8_t* aux = helper ? smem + warp * Epi::AUX : smem + p.off_aux + ow * Epi::AUX;   // helpers: the idle ring of raw stages
    if (!helper) {
      if (ot < m_count) scale[ot] = q.rowscale[m_base + ot] * F::ACC_SCALE;
      asm volatile("bar.sync 1, 256;" ::: "memory");
    }
    const size_t slot = (size_t)rbn * p.nb * 128;                     // floats of one segment
    int nseg = 0;
    for (int u = rg.u0; u < rg.u1; ++nseg) {
      int tile, ks0, ks1;
      segment(u, tile, ks0, ks1);
      const bool last = u >= rg.u1, whole = ks0 == 0 && ks1 == nks;
      if (helper && !last) continue;
      auto sync_out = [&] {
        if (Epi::HELP && last) asm volatile("bar.sync 2, %0;" ::"n"((TS_OUT + TS_WORKERS) * 32) : "memory");
        else asm volatile("bar.sync 1, %0;" ::"n"(TS_OUT * 32) : "memory");
      };
      const int sb = nseg & 1;
      const uint8_t* wrow = nullptr;
      uint32_t e = 0u;
      if constexpr (ts_shifts<FMT>()) {
        if (!helper) {
          wrow = row_start(ot >> 7, tile * p.tile_rows + (ot & 127));   // (of the only block, where there is one)
          e = __ldg(wrow);
        }
      }
      // The helpers have not followed the phases of this barrier (a wait could pass one or two segments early): the output warps
      // have, and the barrier that both meet at below is what lets the helpers read.
      if (!helper) wait(SEG_FULL(sb), (uint32_t)(nseg >> 1) & 1u);
      __syncwarp();
      if constexpr (ts_shifts<FMT>())
        if (!helper) back[ot] = ts_pow2(-ts_row_shift<FMT>(e, wrow));
      if constexpr (FMT != F_NVFP4) {
        uint32_t* mk = marks + (nseg & (TS_MARK_RING - 1)) * 8 + ow;
        if (ow < 4 && __any_sync(0xffffffffu, (mk[0] | mk[4]) != 0u)) {   // a warp adds the shares of a quadrant's marked rows
          const int kind = ks0 > 0 ? 0 : (ks1 < nks ? 1 : 2 + sb);
          ts_add_left_out<FMT>(q, q.part + (size_t)(blockIdx.x * 4 + kind) * slot, mk, ow, tile, m_base, m_count, ks0, ks1, lane);
          __syncwarp();
          if (lane == 0) { mk[0] = 0u; mk[4] = 0u; }
        }
      }
      // Also before the ticket of a cut item: thread 0's release covers the shares that the other warps have added by this barrier,
      // none that they add after it.
      if ((Epi::HELP && last) || FMT != F_NVFP4) sync_out();
      TsItem item{tile, m_base, m_count, q.part + (size_t)(blockIdx.x * 4 + 2 + sb) * slot, nullptr, 0, 1};
      bool mine = true;
      if (!whole) {
        const int first = ts_owner(p, rg.ctas, (long long)tile * nks), end = ts_owner(p, rg.ctas, (long long)(tile + 1) * nks - 1);
        unsigned* count = q.count + (size_t)tile * p.groups + rg.grp;
        if (ot == 0) {
          // release: the part of this CTA (its writers were waited for above); acquire: the parts of the others
          unsigned t;
          asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(t) : "l"(count) : "memory");
          if (t == (unsigned)(end - first)) *count = 0u;
          *ticket = t;
        }
        sync_out();
        mine = __all_sync(0xffffffffu, *ticket == (unsigned)(end - first));   // every other part is in
        item.first = q.part + (size_t)((first * p.groups + rg.grp) * 4 + 1) * slot;
        item.rest = q.part + (size_t)(((first + 1) * p.groups + rg.grp) * 4) * slot;
        item.step = (size_t)p.groups * 4 * slot;
        item.parts = end - first + 1;
      }
      if (mine) Epi::template run<ts_shifts<FMT>()>(ea, q, item, scale, back, aux, ow, Epi::HELP && last ? TS_OUT + TS_WORKERS : TS_OUT, lane);
      if (last) break;
      sync_out();                                                     // the ticket and the policy's buffer are free again
      if (lane == 0) mbar_arrive(SEG_EMPTY(sb));
    }
    if (!helper) Epi::tail(ea, q, smem + p.off_aux, ow, lane);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == TS_MMA_WARP) tmem_dealloc(0u, 512u);
}

}  // namespace qx
