// The dense FP8 GeGLU MLP of one or two tokens, in two launches: quantise + gate/up projection + GeGLU, quantise + down projection.
//
// What bounds it.  18 MB of weights, 3 us at the copy rate, and two chains of latencies (tokens, block maxima, weights, MMAs).  As four launches of the
// kernels for larger batches it took 23 us alone and 29 beside the experts, where it was the longer side of a feed-forward layer: the
// projections are 33 and 22 items of 128 weight rows, each 360 and 270 KB through one SM (12 and 10 us), and the two row-wise kernels
// between them take 2.7 and 4.
//   * The sums are those of the other dense kernels, bit by bit: tcgen05.mma over ascending K into one accumulator, tokens on M, weight rows on N.  M is
//     128; the rows behind the tokens' eight are whatever lies behind their tile (always inside FewSmem), and nobody looks at their results.
//     So a token has the same bits in any batch: alone, or among those that verify a draft.
//   * 44 CTAs take 48 rows of the gate and the same 48 of the up projection, 88 CTAs, two an SM, 32 rows of the down projection, and all of K, so that
//     both launches stay on the SMs that a layer leaves to the dense side.  An MMA takes about as long with 96 rows as with 16 (its 128 token rows
//     come from shared memory either way).  Gate rows / down rows of a CTA, us, the MLP of one token alone and a feed-forward layer with it in a graph: 16 / 16 11.6 and
//     29.5 (its 132 and 176 CTAs keep the experts' off most SMs), 16 / 64 12.0 and 26.4, 32 / 32 11.5 and 25.1, 32 / 64 11.2 and 24.7, 48 / 16 12.3 and 25.7,
//     48 / 32 11.65 and 24.4, 48 / 64 11.7 and 24.5.
//   * All weights that fit are asked for at once, a tensor-map copy and a barrier a K block; the second projection's, alone, while the first one still runs.
//   * Every CTA quantises the tokens for itself while its weights are on their way.  The first projection's also make the products, each once.
// Those launches -> these, us: MLP alone, 1 token 22.9 -> 11.7, 2 21.9 -> 11.7; feed-forward layers in a graph, 1 token 31.8 -> 24.6, 2 32.2 -> 27.7.  Beside the
// experts the second launch starts when the first has ended: as a programmatic one its CTAs, waiting, would hold SMs of the experts' (and gain nothing: 24.4 so,
// 24.75 with it).
#include "gv_common.cuh"
#include "gv_dense_rows.cuh"
#include "gv_gemm_parts.cuh"
#include "gv_launchers.h"

namespace gv {

namespace {

constexpr int kFwWarps = 11;                 // that quantise: 8 columns of a token a thread; every fourth one is also epilogue
constexpr int kFwRowThreads = kFwWarps * 32;
constexpr int kFwWeightWarp = kFwWarps, kFwMmaWarp = kFwWarps + 1;
constexpr int kFwThreads = kFwRowThreads + 64;
constexpr int kFwTokenBytes = 8 * kTileKBytes;  // a K block of the tokens: eight rows, the first one or two of which are tokens
constexpr int kFwMmaBytes = 32;                 // K of an MMA
constexpr int kFwMaxSmem = 232448;
static_assert(kHidden == kFwRowThreads * 8 && kDense % kFwMmaBytes == 0 && kHidden % kFwMmaBytes == 0, "whole MMAs");

// kRows: weight rows of a CTA, MMA-N.
template <int kTokens, int kK, int kRows>
struct alignas(1024) FewSmem {
  static constexpr int kBlocks = (kK + kTileKBytes - 1) / kTileKBytes;
  static constexpr int kWeightBytes = kRows * kTileKBytes;
  static constexpr int kFit = (kFwMaxSmem - 4096 - kBlocks * kFwTokenBytes) / kWeightBytes;
  static constexpr int kStages = kFit < kBlocks ? kFit : kBlocks;
  uint8_t x[kBlocks][kFwTokenBytes];
  uint8_t w[kStages][kWeightBytes];
  uint64_t full[kStages], empty[kStages];
  uint64_t acc_full;
  uint32_t tmem_base;
  volatile int abort;
  float maxima[kTokens][kFwWarps];
  // the MMAs read 128 rows from a block of `x`
  static_assert((kBlocks - 1) * kFwTokenBytes + kTileM * kTileKBytes <= kBlocks * kFwTokenBytes + kStages * kWeightBytes, "reads stay inside");
  static_assert(kRows % 16 == 0 && kRows <= 128, "N of an MMA");
};
template <int kTokens, int kK, int kRows>
constexpr size_t few_smem_bytes() { return sizeof(FewSmem<kTokens, kK, kRows>) + 1024; }
template <int kRows> constexpr uint32_t kFwTmemColumns = kRows <= 32 ? 32 : kRows <= 64 ? 64 : 128;

struct FewParams {
  const __nv_bfloat16* input;   // [tokens, 2816], or the products [tokens, 2112]
  uint8_t* codes;
  float* scales;
  __nv_bfloat16* out;
  __nv_bfloat16* products;
  int* status;
  float gate_w_scale, up_w_scale;
  int tokens;
};

// By the MMA warp.
template <int kRows, class Smem>
__device__ __forceinline__ void few_begin(Smem* smem) {
  tmem_alloc(&smem->tmem_base, kFwTmemColumns<kRows>);
  tmem_relinquish();
}

// By one thread of the weight warp.
template <class Smem>
__device__ __forceinline__ void few_init(Smem* smem, const CUtensorMap* map) {
  for (int s = 0; s < Smem::kStages; ++s) {
    mbar_init(&smem->full[s], 1);
    mbar_init(&smem->empty[s], 1);
  }
  mbar_init(&smem->acc_full, 1);
  smem->abort = 0;
  fence_barrier_init();
  prefetch_tensor_map(map);
}

// K blocks [first, last) of the weights, by one thread of the weight warp; `load` copies a block.
template <class Smem, class Load>
__device__ __forceinline__ void few_fetch(Smem* smem, int first, int last, int* status, Load load) {
#pragma unroll 1
  for (int kb = first; kb < last; ++kb) {
    const int stage = kb % Smem::kStages;
    if (kb >= Smem::kStages && !wait_or_abort(&smem->empty[stage], (kb / Smem::kStages - 1) & 1, smem, status)) return;
    mbar_arrive_expect_tx(&smem->full[stage], Smem::kWeightBytes);
    load(smem->w[stage], &smem->full[stage], kb * kTileKBytes);
  }
}

// All MMAs of the CTA, by one thread, as the K blocks' weights land.
template <int kK, int kRows, class Smem>
__device__ __forceinline__ void few_multiply(Smem* smem, uint32_t tmem_acc, int* status) {
  constexpr int kLast = kK % kTileKBytes ? kK % kTileKBytes / kFwMmaBytes : 4;
  constexpr uint32_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);  // 8 rows x 128 B groups, 128B swizzle
  constexpr uint32_t descriptor = kInstrDescFp8<kRows>;
  const uint32_t x_lo = (smem_u32(smem->x[0]) & 0x3ffffu) >> 4, w_lo = (smem_u32(smem->w[0]) & 0x3ffffu) >> 4;
  tc_fence_after_sync();
#pragma unroll 1
  for (int kb = 0; kb < Smem::kBlocks; ++kb) {
    const int stage = kb % Smem::kStages;
    if (!wait_or_abort(&smem->full[stage], kb / Smem::kStages & 1, smem, status)) {
      // what was asked for lands, and what was issued ends, before shared memory is given up
      for (int b = kb; b < kb + Smem::kStages && b < Smem::kBlocks; ++b)
        mbar_wait_bounded(&smem->full[b % Smem::kStages], b / Smem::kStages & 1, 40000000ll);
      tc_commit(&smem->acc_full);
      mbar_wait_bounded(&smem->acc_full, 0, 40000000ll);
      return;
    }
    const uint32_t a = x_lo + static_cast<uint32_t>(kb) * (kFwTokenBytes >> 4);
    const uint32_t b = w_lo + static_cast<uint32_t>(stage) * (Smem::kWeightBytes >> 4);
    if (kb + 1 < Smem::kBlocks) issue_k_block_fp8<4>(tmem_acc, a, b, hi, descriptor, kb != 0);
    else issue_k_block_fp8<kLast>(tmem_acc, a, b, hi, descriptor, kb != 0);
    if (Smem::kStages < Smem::kBlocks) tc_commit(&smem->empty[stage]);
  }
  tc_commit(&smem->acc_full);
}

// Whether the sums are there, by a warp of the epilogue.
template <class Smem>
__device__ __forceinline__ bool few_sums_there(Smem* smem, int* status) {
  const bool there = __all_sync(0xffffffffu, wait_or_abort(&smem->acc_full, 0, smem, status)) && !smem->abort;
  tc_fence_after_sync();
  return __all_sync(0xffffffffu, there);
}

template <int kRows, class Smem>
__device__ __forceinline__ void few_end(Smem*, uint32_t tmem_acc) {
  tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x >> 5 == kFwMmaWarp) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_acc, kFwTmemColumns<kRows>);
  }
}

// Where eight codes of a token go: 16-byte chunk c of row t at chunk c ^ t of its 128 bytes (128B swizzle).
template <class Smem>
__device__ __forceinline__ void few_store_codes(Smem* smem, int token, int thread, uint2 code) {
  const int column = 8 * thread;
  const int in_block = column % kTileKBytes;
  *reinterpret_cast<uint2*>(smem->x[column / kTileKBytes] + token * kTileKBytes + (((in_block >> 4) ^ token) << 4) + (in_block & 8)) = code;
}

// Scale of a token from the threads' maxima: of all columns, by every thread for itself.
template <class Smem>
__device__ __forceinline__ void few_maximum(Smem* smem, int token, float maximum) {
#pragma unroll
  for (int offset = 16; offset; offset >>= 1) maximum = fmaxf(maximum, __shfl_xor_sync(0xffffffffu, maximum, offset));
  if ((threadIdx.x & 31) == 0) smem->maxima[token][threadIdx.x >> 5] = maximum;
}
template <class Smem>
__device__ __forceinline__ float few_scale(const Smem* smem, int token) {
  float maximum = smem->maxima[token][0];
#pragma unroll
  for (int w = 1; w < kFwWarps; ++w) maximum = fmaxf(maximum, smem->maxima[token][w]);
  return e4m3_row_scale(maximum);
}

// Maxima, scales and codes of the tokens, `raw` being the thread's eight columns of each, into shared memory; CTA 0 also keeps them in
// global memory.  By the first kFwWarps warps; the arithmetic of fp8_quantize_rows_kernel and gelu_quantize_fp8_kernel.
template <int kTokens, int kK, class Smem>
__device__ __forceinline__ void few_quantise(Smem* smem, const uint4 (&raw)[kTokens], const FewParams& p) {
  const int thread = threadIdx.x;
#pragma unroll
  for (int t = 0; t < kTokens; ++t) {
    float x[8], maximum = 0.0f;
    unpack8(raw[t], x);
#pragma unroll
    for (int i = 0; i < 8; ++i) maximum = fmaxf(maximum, fabsf(x[i]));
    few_maximum(smem, t, maximum);
  }
  named_barrier(1, kFwRowThreads);
  if (thread >= kK / 8) return;
#pragma unroll
  for (int t = 0; t < kTokens; ++t) {
    float x[8];
    unpack8(raw[t], x);
    const float scale = few_scale(smem, t);
    const uint2 code = encode_e4m3x8(x, __fdiv_rn(1.0f, scale));
    few_store_codes(smem, t, thread, code);
    if (blockIdx.x == 0 && t < p.tokens) {
      reinterpret_cast<uint2*>(p.codes + static_cast<size_t>(t) * kK)[thread] = code;
      if (thread == 0) p.scales[t] = scale;
    }
  }
  fence_proxy_async_smem();  // the MMAs read the codes
}

// kUnits units of 16 rows of the gate and the same of the up projection, and their GeGLU products.
template <int kTokens, int kUnits>
__global__ void __launch_bounds__(kFwThreads, 1)
dense_few_gate_up_kernel(const __grid_constant__ CUtensorMap map, const FewParams p) {
  constexpr int kRows = 32 * kUnits;
  using Smem = FewSmem<kTokens, kHidden, kRows>;
  extern __shared__ uint8_t smem_raw[];
  Smem* smem = reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int column0 = static_cast<int>(blockIdx.x) * 16 * kUnits;
  if (warp == kFwMmaWarp) few_begin<kRows>(smem);
  if (warp == kFwWeightWarp && lane == 0) few_init(smem, &map);
  grid_dependency_wait();
  grid_launch_dependents();  // after the wait: whoever starts now may read what came before this kernel
  const auto load = [&](void* to, uint64_t* bar, int x) { tma_load_3d(to, &map, bar, x, column0, 0, read_once_policy()); };
  if (warp == kFwWeightWarp) {
    if (lane == 0) few_fetch(smem, 0, Smem::kStages, p.status, load);
    __syncwarp();
  } else if (warp < kFwWarps) {
    uint4 raw[kTokens];
#pragma unroll
    for (int t = 0; t < kTokens; ++t)
      raw[t] = t < p.tokens ? __ldg(reinterpret_cast<const uint4*>(p.input + static_cast<size_t>(t) * kHidden) + threadIdx.x) : uint4{};
    few_quantise<kTokens, kHidden>(smem, raw, p);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_acc = smem->tmem_base;
  if (warp == kFwWeightWarp) {
    if (lane == 0) few_fetch(smem, Smem::kStages, Smem::kBlocks, p.status, load);
    __syncwarp();
  } else if (warp == kFwMmaWarp) {
    if (elect_one()) few_multiply<kHidden, kRows>(smem, tmem_acc, p.status);
    __syncwarp();
  } else if ((warp & 3) == 0 && warp / 4 < kUnits && few_sums_there(smem, p.status)) {
    // tensor-memory lane = token; a unit a warp, every product by a lane of its own
    const int unit = warp / 4;
    uint32_t gates[16], ups[16];
    tmem_load_32x16(tmem_acc + unit * 16, gates);
    tmem_load_32x16(tmem_acc + (kUnits + unit) * 16, ups);
    tmem_load_wait(gates, ups);
    const int token = lane >> 4, row = lane & 15;
    uint32_t gate_bits = 0, up_bits = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const uint32_t g = __shfl_sync(0xffffffffu, gates[i], token), u = __shfl_sync(0xffffffffu, ups[i], token);
      if (i == row) {
        gate_bits = g;
        up_bits = u;
      }
    }
    if (token < p.tokens) {
      const __nv_bfloat16 gate = __float2bfloat16_rn(__uint_as_float(gate_bits)), up = __float2bfloat16_rn(__uint_as_float(up_bits));
      const int column = column0 + unit * 16 + row;
      p.out[static_cast<size_t>(token) * (2 * kDense) + column] = gate;
      p.out[static_cast<size_t>(token) * (2 * kDense) + kDense + column] = up;
      const float scale = few_scale(smem, token);
      p.products[token * kDense + column] =
          __float2bfloat16_rn(geglu_tanh(__bfloat162float(gate), __bfloat162float(up), __fmul_rn(scale, p.gate_w_scale), __fmul_rn(scale, p.up_w_scale)));
    }
  }
  few_end<kRows>(smem, tmem_acc);
}

// The products' quantisation and kRows rows of the down projection, likewise.
template <int kTokens, int kRows>
__global__ void __launch_bounds__(kFwThreads, 1)
dense_few_down_kernel(const __grid_constant__ CUtensorMap map, const FewParams p) {
  using Smem = FewSmem<kTokens, kDense, kRows>;
  static_assert(Smem::kStages == Smem::kBlocks, "every block has a place");
  extern __shared__ uint8_t smem_raw[];
  Smem* smem = reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = static_cast<int>(blockIdx.x) * kRows;
  if (warp == kFwMmaWarp) few_begin<kRows>(smem);
  if (warp == kFwWeightWarp) {
    // The first projection lets this kernel start after its own wait: the weights come from before it.
    // (a box that reaches past the rows' end is filled up with zeros)
    if (lane == 0) {
      few_init(smem, &map);
      few_fetch(smem, 0, Smem::kBlocks, p.status,
                [&](void* to, uint64_t* bar, int x) { tma_load_2d(to, &map, bar, x, row0, read_once_policy()); });
    }
    __syncwarp();
  }
  grid_dependency_wait();
  grid_launch_dependents();
  if (warp < kFwWarps) {
    uint4 raw[kTokens];
#pragma unroll
    for (int t = 0; t < kTokens; ++t)
      raw[t] = threadIdx.x < kDense / 8 && t < p.tokens ? reinterpret_cast<const uint4*>(p.input + t * kDense)[threadIdx.x] : uint4{};
    few_quantise<kTokens, kDense>(smem, raw, p);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_acc = smem->tmem_base;
  if (warp == kFwMmaWarp) {
    if (elect_one()) few_multiply<kDense, kRows>(smem, tmem_acc, p.status);
    __syncwarp();
  } else if ((warp & 3) == 0 && warp < kFwWarps && warp / 4 < kRows / 16 && few_sums_there(smem, p.status)) {
    constexpr int kEpilogueWarps = (kFwWarps + 3) / 4;
#pragma unroll 1
    for (int chunk = warp / 4; chunk < kRows / 16; chunk += kEpilogueWarps) {
      uint32_t r[16];  // of token `lane`
      tmem_load_32x16(tmem_acc + chunk * 16, r);
      tmem_load_wait(r);
      if (lane < p.tokens) {
        uint4* out = reinterpret_cast<uint4*>(p.out + static_cast<size_t>(lane) * kHidden + row0 + chunk * 16);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t pairs[4];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            pairs[i] = pack_bf16x2(__uint_as_float(r[8 * half + 2 * i]), __uint_as_float(r[8 * half + 2 * i + 1]));
          out[half] = make_uint4(pairs[0], pairs[1], pairs[2], pairs[3]);
        }
      }
      __syncwarp();
    }
  }
  few_end<kRows>(smem, tmem_acc);
}

static_assert(kDenseFewTokens == 2, "variants");
constexpr int kFwUnits = kDenseFewUpRows / 16;
static_assert(kDenseFewUpRows % 16 == 0 && kDense % kDenseFewUpRows == 0 && kHidden % kDenseFewDownRows == 0, "whole CTAs");

template <int kTokens> constexpr size_t few_up_bytes() { return few_smem_bytes<kTokens, kHidden, 2 * kDenseFewUpRows>(); }
template <int kTokens> constexpr size_t few_down_bytes() { return few_smem_bytes<kTokens, kDense, kDenseFewDownRows>(); }
static_assert(few_up_bytes<kDenseFewTokens>() <= kFwMaxSmem && few_down_bytes<kDenseFewTokens>() <= kFwMaxSmem, "shared memory of a CTA");

template <int kTokens>
cudaError_t prepare() {
  const cudaError_t e = cudaFuncSetAttribute(dense_few_gate_up_kernel<kTokens, kFwUnits>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(few_up_bytes<kTokens>()));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(dense_few_down_kernel<kTokens, kDenseFewDownRows>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(few_down_bytes<kTokens>()));
}

template <int kTokens>
void launch(const DenseFewOperands& op, int tokens, cudaStream_t stream) {
  FewParams up{};
  up.input = static_cast<const __nv_bfloat16*>(op.input);
  up.codes = op.act_codes;
  up.scales = op.act_scales;
  up.out = static_cast<__nv_bfloat16*>(op.gate_up);
  up.products = static_cast<__nv_bfloat16*>(op.products);
  up.status = op.status;
  up.gate_w_scale = op.gate_scale;
  up.up_w_scale = op.up_scale;
  up.tokens = tokens;
  launch_chained(dense_few_gate_up_kernel<kTokens, kFwUnits>, dim3(kDense / kDenseFewUpRows), dim3(kFwThreads), few_up_bytes<kTokens>(), stream,
                 *op.map_gate_up, up);
  FewParams down{};
  down.input = up.products;
  down.codes = op.prod_codes;
  down.scales = op.prod_scales;
  down.out = static_cast<__nv_bfloat16*>(op.out);
  down.status = op.status;
  down.tokens = tokens;
  if (op.serial_launch)
    dense_few_down_kernel<kTokens, kDenseFewDownRows><<<kHidden / kDenseFewDownRows, kFwThreads, few_down_bytes<kTokens>(), stream>>>(*op.map_down, down);
  else
    launch_chained(dense_few_down_kernel<kTokens, kDenseFewDownRows>, dim3(kHidden / kDenseFewDownRows), dim3(kFwThreads), few_down_bytes<kTokens>(), stream,
                   *op.map_down, down);
}

}  // namespace

int prepare_dense_few() {
  cudaError_t e = prepare<1>();
  if (e == cudaSuccess) e = prepare<2>();
  return static_cast<int>(e);
}

void launch_dense_few(const DenseFewOperands& op, int tokens, cudaStream_t stream) {
  if (tokens == 1) launch<1>(op, tokens, stream);
  else launch<2>(op, tokens, stream);
}

}  // namespace gv
