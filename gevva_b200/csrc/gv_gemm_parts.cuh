// Pieces shared by the grouped GEMM kernels (grouped_gemm.cu: one CTA per tile;
// grouped_gemm_pair.cu: a CTA pair per tile pair): the launch parameters, the epilogue arithmetic
// and the shared-memory staged store.
#pragma once

#include "gv_common.cuh"
#include "gv_launchers.h"

namespace gv {
namespace {

constexpr int kEpilogueWarpsPerQuarter = 4;  // each takes a quarter of a tile's columns
constexpr int kEpilogueThreads = 4 * kEpilogueWarpsPerQuarter * 32;
constexpr int kStoreColumns = 128;                        // columns per store pass (plain epilogue)
constexpr int kStageRowBytes = kStoreColumns * 2;         // one bf16 row of a store pass
constexpr int kStagingBytesPerWarp = 32 * kStageRowBytes; // 8 KiB

enum GemmMode { kPlain = 0, kGeglu = 1, kFp8 = 2 };  // kFp8: dense E4M3 operands, plain epilogue


struct GemmParams {
  const uint8_t* a_scales;
  const uint8_t* b_scales;   // kPlain: sidecar layout; kGeglu: re-tiled copy
  const float* alpha;
  __nv_bfloat16* out;        // kPlain
  const unsigned long long* row_dest;  // kPlain, optional: address of each output row (may be peer memory)
  uint8_t* next_codes;       // kGeglu: w2 operand codes [rows, 352]
  uint8_t* next_scales;      // kGeglu: w2 operand scale regions
  const float* next_scale_q; // kGeglu: g2.input_scale_quant [128]
  const int* tile_expert;
  const int* expert_offsets;
  const int* scale_row_offsets;
  const int* num_m_tiles;
  const int* tile_first;     // optional: first row tile of this launch
  int* status;
  int n_out;
  int n_tiles;      // work items per row tile
  int groups;       // k_in / 16
  int k_blocks;     // ceil(k_in / 256)
  int last_mmas;    // MMAs (K = 64 each) in the last K block, 1..4
  bool early_weights;  // see GemmOperands
};

// One 128-byte K block of the dense FP8 projections: kMmas MMAs of K = 32 E4M3 elements (32 bytes, a descriptor step of 2), no scale
// factors.  Instruction descriptor: fp32 accumulate (bit 4), E4M3 x E4M3 (format 0), both K-major, N at [17,23) in units of 8, M at [24,29) in units of 16.
template <int kN>
constexpr uint32_t kInstrDescFp8 = (1u << 4) | (static_cast<uint32_t>(kN >> 3) << 17) |
                                   (static_cast<uint32_t>(kTileM >> 4) << 24);

template <int kMmas>
__device__ __forceinline__ void issue_k_block_fp8(uint32_t tmem_acc, uint32_t a_lo, uint32_t b_lo,
                                                  uint32_t hi_ab, uint32_t descriptor, uint32_t accumulate) {
#define GV_MMA8(j, pred)                                                   \
  "add.u32 lo, %1, " #j "*2;\n\t"                                          \
  "mov.b64 d0, {lo, %3};\n\t"                                              \
  "add.u32 lo, %2, " #j "*2;\n\t"                                          \
  "mov.b64 d1, {lo, %3};\n\t"                                              \
  "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], d0, d1, %4, " pred ";\n\t"
#define GV_OPERANDS8 ::"r"(tmem_acc), "r"(a_lo), "r"(b_lo), "r"(hi_ab), "r"(descriptor), "r"(accumulate) : "memory"
#define GV_PROLOGUE8 "{\n\t.reg .pred p, pt;\n\t.reg .b32 lo;\n\t.reg .b64 d0, d1;\n\t" \
                     "setp.ne.b32 p, %5, 0;\n\tsetp.eq.b32 pt, 0, 0;\n\t"
  asm volatile(GV_PROLOGUE8 GV_MMA8(0, "p") "}" GV_OPERANDS8);
  if constexpr (kMmas >= 2) asm volatile(GV_PROLOGUE8 GV_MMA8(1, "pt") "}" GV_OPERANDS8);
  if constexpr (kMmas >= 3) asm volatile(GV_PROLOGUE8 GV_MMA8(2, "pt") "}" GV_OPERANDS8);
  if constexpr (kMmas >= 4) asm volatile(GV_PROLOGUE8 GV_MMA8(3, "pt") "}" GV_OPERANDS8);
#undef GV_MMA8
#undef GV_OPERANDS8
#undef GV_PROLOGUE8
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  const __nv_bfloat162 pair = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&pair);
}

// bf16 rounding of alpha*acc, returned as float: the value the reference's GEMM
// epilogue stores and its GeGLU kernel reads back (src/nvfp4_cutlass.cu:582-583).
__device__ __forceinline__ float round_through_bf16(float alpha, uint32_t acc_bits) {
  return __bfloat162float(__float2bfloat16_rn(__fmul_rn(alpha, __uint_as_float(acc_bits))));
}

// Plain epilogue, one store pass: this warp's 32 rows x 32 columns (already scaled and
// rounded) go to the quarter's staging tile (32 rows x 256 bytes), then the four warps of the
// quarter write the tile out so that every store instruction covers two full 256-byte row
// segments.  16-byte chunk c of row r lives at chunk position c ^ (r & 15), which keeps the
// row-wise writes and the two-rows-per-instruction reads at the minimum number of bank passes.
__device__ __forceinline__ void stage_and_store(const uint32_t (&r)[32], float alpha, uint8_t* staging,
                                                int quarter, int sub, int lane, int rows_valid,
                                                int row0, int column0, const GemmParams& p) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint4 v;
    v.x = pack_bf16x2(__fmul_rn(alpha, __uint_as_float(r[8 * i])),
                      __fmul_rn(alpha, __uint_as_float(r[8 * i + 1])));
    v.y = pack_bf16x2(__fmul_rn(alpha, __uint_as_float(r[8 * i + 2])),
                      __fmul_rn(alpha, __uint_as_float(r[8 * i + 3])));
    v.z = pack_bf16x2(__fmul_rn(alpha, __uint_as_float(r[8 * i + 4])),
                      __fmul_rn(alpha, __uint_as_float(r[8 * i + 5])));
    v.w = pack_bf16x2(__fmul_rn(alpha, __uint_as_float(r[8 * i + 6])),
                      __fmul_rn(alpha, __uint_as_float(r[8 * i + 7])));
    const int c = sub * 4 + i;
    *reinterpret_cast<uint4*>(staging + lane * kStageRowBytes + ((c ^ (lane & 15)) << 4)) = v;
  }
  named_barrier(1 + quarter, kEpilogueWarpsPerQuarter * 32);
  unsigned long long keep_in_l2;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(keep_in_l2));
  const int c = lane & 15;
  __nv_bfloat16* dst = p.out + static_cast<size_t>(row0 + quarter * 32) * p.n_out + column0 + c * 8;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r2 = 2 * (sub * 4 + i) + (lane >> 4);
    const uint4 v = *reinterpret_cast<const uint4*>(staging + r2 * kStageRowBytes + ((c ^ (r2 & 15)) << 4));
    if (quarter * 32 + r2 < rows_valid) {
      if (p.row_dest) {
        // expert-parallel combine: the row goes straight to its source rank's buffer
        __nv_bfloat16* remote = reinterpret_cast<__nv_bfloat16*>(p.row_dest[row0 + quarter * 32 + r2]);
        *reinterpret_cast<uint4*>(remote + column0 + c * 8) = v;
      } else {
        // The rows are read back by the weighted reduce (or the next stage) right after this
        // launch: ask L2 to keep them (without the hint the reduce finds 2 % of them there).
        asm volatile("st.global.L2::cache_hint.v4.b32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(
                         dst + static_cast<size_t>(r2) * p.n_out),
                     "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "l"(keep_in_l2)
                     : "memory");
      }
    }
  }
  named_barrier(1 + quarter, kEpilogueWarpsPerQuarter * 32);  // staging is rewritten next pass
}

// Fused epilogue arithmetic for one 16-value block of one row.
__device__ __forceinline__ uint32_t geglu_block(const uint32_t (&up)[16], const uint32_t (&gate)[16],
                                                float alpha, float multiplier, const float* erf_table,
                                                uint32_t& codes_lo, uint32_t& codes_hi) {
  float values[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float g = round_through_bf16(alpha, gate[i]);
    const float u = round_through_bf16(alpha, up[i]);
    values[i] = __fmul_rn(gv_gelu_erf(g, erf_table), u);
  }
  return quantize_block16(values, multiplier, codes_lo, codes_hi);
}

// The same arithmetic in a third of the instructions, for the kernels that keep its tables.
//
// At FP4 rates the GELU and quantisation of one output value cost as many issue slots as its 5632
// multiply-adds cost tensor cycles, so what a value costs matters: 24 instructions of erf (two of
// them conversions at a quarter of the rate, two 16-byte table loads that take seven shared-memory
// wavefronts each) become one 4-byte load.  That works because the gate has been rounded to bf16: erf's
// argument takes a few thousand values, and `erf_of` holds gv_erff for every bf16 magnitude from 2^-14 up
// to where it is 1.  Smaller magnitudes (one gate in 20000 of unit variance) send the whole block
// through the polynomial.  The results are gv_gelu_erf's and quantize_block16's, bit for bit.
constexpr int kErfFirst = (127 - 14) << 7;                    // bf16 bits of 2^-14
constexpr int kErfEntries = 16 * 128 + 54 + 2;                // up to 4 * sqrt(2), where |x| / sqrt(2) >= 4 and erf is 1

struct GegluTables {
  float erf_of[kErfEntries];
  alignas(16) float reciprocals[GV_RECIPROCAL_FLOATS];
  alignas(16) float erf_table[GV_ERF_TABLE_FLOATS];
};
static __constant__ float g_reciprocals[GV_RECIPROCAL_FLOATS] = GV_RECIPROCALS_INIT;

// Two steps with a block barrier after each (the second reads what the first wrote).
__device__ __forceinline__ void load_geglu_tables(GegluTables* tables) {
  load_erf_table(tables->erf_table);
  if (threadIdx.x < GV_RECIPROCAL_FLOATS) tables->reciprocals[threadIdx.x] = g_reciprocals[threadIdx.x];
}
__device__ __forceinline__ void fill_geglu_tables(GegluTables* tables) {
  for (int i = threadIdx.x; i < kErfEntries; i += blockDim.x)
    tables->erf_of[i] = gv_erff(__fmul_rn(__uint_as_float(static_cast<uint32_t>(kErfFirst + i) << 16), 0.7071067811865475f),
                                tables->erf_table);
}

// gv_erff of a bf16 magnitude below the table over the square root of two: its first interval, whose coefficients are the same for all lanes.
__device__ __forceinline__ float erf_below_table(float magnitude) {
  const float u = __fsub_rn(__fmul_rn(magnitude, 0.7071067811865475f), 0.25f);
  float p = g_erf_table[0][6];
#pragma unroll
  for (int i = 5; i >= 0; --i) p = __fmaf_rn(p, u, g_erf_table[0][i]);
  return p;
}

// erf-GELU of a bf16 value from erf of its magnitude (gv_gelu_erf's last three operations).
__device__ __forceinline__ float gelu_from_erf(float value, float erf_of_magnitude) {
  return __fmul_rn(__fmul_rn(0.5f, value), __fadd_rn(1.0f, copysignf(erf_of_magnitude, value)));
}

// Index of a bf16 magnitude (15 bits) in erf_of; negative where the table does not reach.
__device__ __forceinline__ int erf_index(uint32_t magnitude) {
  return min(static_cast<int>(magnitude) - kErfFirst, kErfEntries - 1);
}

__device__ __forceinline__ float gelu_of_bf16(float value, const GegluTables* tables) {
  const int index = erf_index((__float_as_uint(value) >> 16) & 0x7fffu);
  return index >= 0 ? gelu_from_erf(value, tables->erf_of[index]) : gv_gelu_erf(value, tables->erf_table);
}

// quantize_block16 with the divisions of gv_exact.h.
__device__ __forceinline__ uint32_t quantize_block16_fast(const float (&values)[16], float multiplier,
                                                          const float* reciprocals, uint32_t& codes_lo,
                                                          uint32_t& codes_hi) {
  float maximum = 0.0f;
#pragma unroll
  for (int i = 0; i < 16; ++i) maximum = fmaxf(maximum, fabsf(values[i]));
  const uint32_t scale = encode_e4m3(gv_sixth(__fmul_rn(multiplier, maximum)));
  const float inverse = gv_scale_inverse_exact(multiplier) ? gv_scale_inverse(multiplier, scale, reciprocals)
                                                           : scale_inverse_divided(multiplier, scale);
  uint32_t words[2];
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const float* v = values + 8 * half;
    asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
        "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
        : "=r"(words[half])
        : "f"(__fmul_rn(v[0], inverse)), "f"(__fmul_rn(v[1], inverse)), "f"(__fmul_rn(v[2], inverse)),
          "f"(__fmul_rn(v[3], inverse)), "f"(__fmul_rn(v[4], inverse)), "f"(__fmul_rn(v[5], inverse)),
          "f"(__fmul_rn(v[6], inverse)), "f"(__fmul_rn(v[7], inverse)));
  }
  codes_lo = words[0];
  codes_hi = words[1];
  return scale;
}

// One 16-value block from up and gate values already rounded to bf16, two to a word.
__device__ __forceinline__ uint32_t geglu_block_of_bf16(const uint32_t (&ups)[8], const uint32_t (&gates)[8],
                                                        float multiplier, const GegluTables* tables,
                                                        uint32_t& codes_lo, uint32_t& codes_hi) {
  int smallest = 0;  // its sign bit: some magnitude lies below the table
#pragma unroll
  for (int i = 0; i < 8; ++i)
    smallest |= (static_cast<int>(gates[i] & 0x7fffu) - kErfFirst) | (static_cast<int>((gates[i] >> 16) & 0x7fffu) - kErfFirst);
  float values[16];
  if (smallest >= 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      values[2 * i] = gelu_from_erf(__uint_as_float(gates[i] << 16), tables->erf_of[erf_index(gates[i] & 0x7fffu)]);
      values[2 * i + 1] =
          gelu_from_erf(__uint_as_float(gates[i] & 0xffff0000u), tables->erf_of[erf_index((gates[i] >> 16) & 0x7fffu)]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      values[2 * i] = gv_gelu_erf(__uint_as_float(gates[i] << 16), tables->erf_table);
      values[2 * i + 1] = gv_gelu_erf(__uint_as_float(gates[i] & 0xffff0000u), tables->erf_table);
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    values[2 * i] = __fmul_rn(values[2 * i], __uint_as_float(ups[i] << 16));
    values[2 * i + 1] = __fmul_rn(values[2 * i + 1], __uint_as_float(ups[i] & 0xffff0000u));
  }
  return quantize_block16_fast(values, multiplier, tables->reciprocals, codes_lo, codes_hi);
}

// One 16-value block of one row from the accumulators.
__device__ __forceinline__ uint32_t geglu_block_fast(const uint32_t (&up)[16], const uint32_t (&gate)[16], float alpha,
                                                     float multiplier, const GegluTables* tables, uint32_t& codes_lo,
                                                     uint32_t& codes_hi) {
  uint32_t gates[8], ups[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    gates[i] = pack_bf16x2(__fmul_rn(alpha, __uint_as_float(gate[2 * i])), __fmul_rn(alpha, __uint_as_float(gate[2 * i + 1])));
    ups[i] = pack_bf16x2(__fmul_rn(alpha, __uint_as_float(up[2 * i])), __fmul_rn(alpha, __uint_as_float(up[2 * i + 1])));
  }
  return geglu_block_of_bf16(ups, gates, multiplier, tables, codes_lo, codes_hi);
}

constexpr int kFusedItems = (kInter + 127) / 128;  // 6
// w13 scales re-tiled by unit of 64 intermediate columns (64 up rows, 64 gate rows): [expert][unit][K block
// of 256][2 KiB]; the twelfth unit of an expert pads it to pairs.
constexpr int kUnits = kInter / 64;                // 11
constexpr int kUnitSlots = kUnits + 1;


// Instruction descriptor: E2M1 x E2M1 (format 1 in the mxf4 kinds), both K-major,
// UE4M3 scales (bit 23 clear), N at [17,23) in units of 8, M at [24,29) in units of 16,
// K = 64 (bit 31 clear), scale ids 0.
template <int kN>
constexpr uint32_t kInstrDesc = (1u << 7) | (1u << 10) | (static_cast<uint32_t>(kN >> 3) << 17) |
                                (static_cast<uint32_t>(kTileM >> 4) << 24);

// One K block's worth of tensor-core work, issued by two threads.  The scale copier issues
// kMmas scale-factor atom copies per operand half (shared -> tensor memory, issue_sf_copies); the
// MMA thread, once those have landed, issues kMmas MMAs of K = 64 (issue_mmas).  Everything is
// derived from 32-bit descriptor bases with immediate offsets so that an issuing thread spends
// a handful of integer instructions per tcgen05 instruction.
//   a_lo / b_lo     low words of the operand descriptors of this stage (address >> 4)
//   sfa_lo / sfb_lo low words of the scale-factor descriptors of this stage
//   hi_ab / hi_sf   high words (stride, version, swizzle) shared by all stages
// Scale columns of a K block in tensor memory: at N = 128, A of MMA j at +4j and B at +16+4j;
// at N = 256, A at +16j, B rows 0..127 at +16j+4, B rows 128..255 at +16j+8 (the second half of
// the weight scales lies 2 KiB = 128 descriptor units after the first in shared memory).  kHalf: the
// N = 256 layout with only its first 128 weight rows present, for half the tensor time.
template <int kMmas, int kN, bool kHalf = false>
__device__ __forceinline__ void issue_sf_copies(uint32_t tmem_sf, uint32_t sfa_lo, uint32_t sfb_lo, uint32_t hi_sf) {
  static_assert(kMmas >= 1 && kMmas <= 4, "a K block holds one to four MMAs");
#define GV_SF_OPERANDS ::"r"(tmem_sf), "r"(sfa_lo), "r"(sfb_lo), "r"(hi_sf) : "memory"
#define GV_SF_PROLOGUE "{\n\t.reg .b32 lo, ta;\n\t.reg .b64 d0;\n\t"
#define GV_SF_ONE(source, source_offset, column)                             \
  "add.u32 lo, " source ", " source_offset ";\n\t"                           \
  "mov.b64 d0, {lo, %3};\n\t"                                                \
  "add.u32 ta, %0, " column ";\n\t"                                          \
  "tcgen05.cp.cta_group::1.32x128b.warpx4 [ta], d0;\n\t"
  if constexpr (kN == 128) {
#define GV_SF_COPY(j) GV_SF_ONE("%1", #j "*32", #j "*4") GV_SF_ONE("%2", #j "*32", "16+" #j "*4")
    asm volatile(GV_SF_PROLOGUE GV_SF_COPY(0) "}" GV_SF_OPERANDS);
    if constexpr (kMmas >= 2) asm volatile(GV_SF_PROLOGUE GV_SF_COPY(1) "}" GV_SF_OPERANDS);
    if constexpr (kMmas >= 3) asm volatile(GV_SF_PROLOGUE GV_SF_COPY(2) "}" GV_SF_OPERANDS);
    if constexpr (kMmas >= 4) asm volatile(GV_SF_PROLOGUE GV_SF_COPY(3) "}" GV_SF_OPERANDS);
#undef GV_SF_COPY
  } else {
#define GV_SF_COPY(j) GV_SF_ONE("%1", #j "*32", #j "*16") GV_SF_ONE("%2", #j "*32", "4+" #j "*16")
    asm volatile(GV_SF_PROLOGUE GV_SF_COPY(0) "}" GV_SF_OPERANDS);
    if constexpr (kMmas >= 2) asm volatile(GV_SF_PROLOGUE GV_SF_COPY(1) "}" GV_SF_OPERANDS);
    if constexpr (kMmas >= 3) asm volatile(GV_SF_PROLOGUE GV_SF_COPY(2) "}" GV_SF_OPERANDS);
    if constexpr (kMmas >= 4) asm volatile(GV_SF_PROLOGUE GV_SF_COPY(3) "}" GV_SF_OPERANDS);
#undef GV_SF_COPY
    if constexpr (!kHalf) {
#define GV_SF_COPY(j) GV_SF_ONE("%2", "128+" #j "*32", "8+" #j "*16")
      asm volatile(GV_SF_PROLOGUE GV_SF_COPY(0) "}" GV_SF_OPERANDS);
      if constexpr (kMmas >= 2) asm volatile(GV_SF_PROLOGUE GV_SF_COPY(1) "}" GV_SF_OPERANDS);
      if constexpr (kMmas >= 3) asm volatile(GV_SF_PROLOGUE GV_SF_COPY(2) "}" GV_SF_OPERANDS);
      if constexpr (kMmas >= 4) asm volatile(GV_SF_PROLOGUE GV_SF_COPY(3) "}" GV_SF_OPERANDS);
#undef GV_SF_COPY
    }
  }
#undef GV_SF_ONE
#undef GV_SF_PROLOGUE
#undef GV_SF_OPERANDS
}

template <int kMmas, int kN, bool kHalf = false>
__device__ __forceinline__ void issue_mmas(uint32_t tmem_acc, uint32_t tmem_sf, uint32_t a_lo, uint32_t b_lo,
                                           uint32_t hi_ab, uint32_t accumulate) {
  static_assert(kMmas >= 1 && kMmas <= 4, "a K block holds one to four MMAs");
#define GV_OPERANDS                                                                                  \
  ::"r"(tmem_acc), "r"(tmem_sf), "r"(a_lo), "r"(b_lo), "r"(hi_ab), "r"(kInstrDesc<kHalf ? kN / 2 : kN>), "r"(accumulate) \
  : "memory"
#define GV_PROLOGUE "{\n\t.reg .pred p, pt;\n\t.reg .b32 lo, ta, tb;\n\t.reg .b64 d0, d1;\n\t" \
                    "setp.ne.b32 p, %6, 0;\n\tsetp.eq.b32 pt, 0, 0;\n\t"
#define GV_MMA(j, step, sfb_column, pred)                                  \
  "add.u32 lo, %2, " #j "*2;\n\t"                                          \
  "mov.b64 d0, {lo, %4};\n\t"                                              \
  "add.u32 lo, %3, " #j "*2;\n\t"                                          \
  "mov.b64 d1, {lo, %4};\n\t"                                              \
  "add.u32 ta, %1, " #j "*" #step ";\n\t"                                  \
  "add.u32 tb, %1, " #j "*" #step "+" #sfb_column ";\n\t"                  \
  "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X"      \
  " [%0], d0, d1, %5, [ta], [tb], " pred ";\n\t"
  if constexpr (kN == 128) {
    asm volatile(GV_PROLOGUE GV_MMA(0, 4, 16, "p") "}" GV_OPERANDS);
    if constexpr (kMmas >= 2) asm volatile(GV_PROLOGUE GV_MMA(1, 4, 16, "pt") "}" GV_OPERANDS);
    if constexpr (kMmas >= 3) asm volatile(GV_PROLOGUE GV_MMA(2, 4, 16, "pt") "}" GV_OPERANDS);
    if constexpr (kMmas >= 4) asm volatile(GV_PROLOGUE GV_MMA(3, 4, 16, "pt") "}" GV_OPERANDS);
  } else {
    asm volatile(GV_PROLOGUE GV_MMA(0, 16, 4, "p") "}" GV_OPERANDS);
    if constexpr (kMmas >= 2) asm volatile(GV_PROLOGUE GV_MMA(1, 16, 4, "pt") "}" GV_OPERANDS);
    if constexpr (kMmas >= 3) asm volatile(GV_PROLOGUE GV_MMA(2, 16, 4, "pt") "}" GV_OPERANDS);
    if constexpr (kMmas >= 4) asm volatile(GV_PROLOGUE GV_MMA(3, 16, 4, "pt") "}" GV_OPERANDS);
  }
#undef GV_MMA
#undef GV_OPERANDS
#undef GV_PROLOGUE
}


}  // namespace
}  // namespace gv
