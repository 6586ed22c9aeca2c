// The dense FP8 GeGLU MLP of one or two tokens, in two launches: quantise + gate/up projection + GeGLU, quantise + down projection.
//
// What bounds it.  18 MB of weights, 3 us at the copy rate, and two chains of latencies (tokens, block maxima, weights, sums).  As four launches of the
// kernels for larger batches it took 23 us alone and 29 beside the experts, where it was the longer side of a feed-forward layer: the
// projections are 33 and 22 items of 128 weight rows, each 360 and 270 KB through one SM (12 and 10 us), and the two row-wise kernels
// between them take 2.7 and 4.
//   * A CTA takes 16 weight rows and all of K, an eleventh for each of its warps: 264 and 176 CTAs.  All bytes of a lane (eight or six
//     16-byte loads) are asked for at once, the second projection's, alone, while the first one still runs.
//   * Every CTA quantises the tokens for itself while its weights are on their way.  The first projection's have eight gate rows and the same
//     up rows, so that each product is made once (with all of them made by every CTA of the second: 11.1 us at one token, 17 at four).
//   * E4M3 values are exact in fp16, and so are the products of two in fp32: mma.m16n8k16 with fp32 sums, the tokens on its N side (a shape
//     that tcgen05 would fill with 128 rows).  A lane's 16 consecutive bytes are four MMAs' share of K for it, in the same order on both
//     sides.  The warps' sums are added in a fixed order.
//     Against sums in 64 bits the projections are as far off as the tcgen05 ones: 1.7e-3 of the norm, all of it the bf16
//     result; 2 to 4 results in ten thousand are not the nearest bf16 (those: 2 to 5).
// MLP alone, us, those launches -> these: 1 token 23.3 -> 8.8, 2 22.5 -> 8.5 (a variant for four tokens 22.4 -> 9.9, for eight 22.5 -> 15: every CTA
// quantises all of them).  Feed-forward layers in a graph, us a layer: 1 token 31.0 -> 25.7, 2 31.5 -> 29.1, 3 32.0 -> 32.4, 4 34.7 -> 35.8, 5 39.8 -> 45
// to 51: the longer these CTAs hold SMs, the later the experts' start, which want them all.  Hence the line at two tokens, and beside the
// experts the second launch starts when the first has ended (as a programmatic one its CTAs, waiting, hold SMs: 2 tokens 29.4 instead of 29.2).
#include <stddef.h>

#include "gv_common.cuh"
#include "gv_launchers.h"

namespace gv {

namespace {

constexpr int kFwWarps = 11;
constexpr int kFwThreads = kFwWarps * 32;    // 352: 8 columns of a token each
constexpr int kFwRows = 16;                  // weight rows of a CTA
constexpr int kFwDense = 2112;
constexpr int kFwStepBytes = 64;             // of a weight row: 16 bytes a lane of a quad
constexpr int kFwRowBytes = kHidden + 16;    // tokens in shared memory, rows in banks of their own
static_assert(kHidden == kFwThreads * 8 && kHidden % (kFwWarps * kFwStepBytes) == 0 && kFwDense % (kFwWarps * kFwStepBytes) == 0, "whole steps for every warp");
static_assert(kFwDense % 8 == 0 && kHidden % kFwRows == 0, "whole CTAs");

template <int kTokens>
struct FewSmem {
  alignas(16) uint8_t x[kTokens][kFwRowBytes];
  float maxima[kTokens][kFwWarps];
  alignas(16) float sums[kFwWarps][kFwRows][8];  // stored two at a time
};
static_assert(offsetof(FewSmem<1>, sums) % 8 == 0 && kFwRowBytes % 16 == 0, "alignment of what is stored and read in pieces");

template <int kSteps>
struct FewWeights {
  uint4 low[kSteps], high[kSteps];  // row lane / 4 and row lane / 4 + 8
};

// `low` and `high`: the CTA's two groups of eight rows.
template <int kSteps>
__device__ __forceinline__ void few_fetch(FewWeights<kSteps>& w, const uint8_t* low, const uint8_t* high) {
  constexpr int k_bytes = kSteps * kFwWarps * kFwStepBytes;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int offset = (lane >> 2) * k_bytes + warp * (kSteps * kFwStepBytes) + (lane & 3) * 16;
  const uint64_t policy = read_once_policy();
#pragma unroll
  for (int s = 0; s < kSteps; ++s) {
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=r"(w.low[s].x), "=r"(w.low[s].y), "=r"(w.low[s].z), "=r"(w.low[s].w)
                 : "l"(low + offset + s * kFwStepBytes), "l"(policy));
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=r"(w.high[s].x), "=r"(w.high[s].y), "=r"(w.high[s].z), "=r"(w.high[s].w)
                 : "l"(high + offset + s * kFwStepBytes), "l"(policy));
  }
}

// Two E4M3 values, the lower byte first, as fp16 (exact).
__device__ __forceinline__ uint32_t few_halves(uint32_t pair16) {
  uint32_t h;
  asm("{\n\t.reg .b16 p;\n\tcvt.u16.u32 p, %1;\n\tcvt.rn.f16x2.e4m3x2 %0, p;\n\t}" : "=r"(h) : "r"(pair16));
  return h;
}

template <int kTokens, int kSteps>
__device__ __forceinline__ void few_multiply(const FewWeights<kSteps>& w, FewSmem<kTokens>* smem) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int token = lane >> 2;
  const uint8_t* x = smem->x[token < kTokens ? token : 0] + warp * (kSteps * kFwStepBytes) + (lane & 3) * 16;
  float acc[4] = {0, 0, 0, 0};
#pragma unroll
  for (int s = 0; s < kSteps; ++s) {
    uint4 b = *reinterpret_cast<const uint4*>(x + s * kFwStepBytes);
    if (token >= kTokens) b = uint4{};
    const uint32_t lows[4] = {w.low[s].x, w.low[s].y, w.low[s].z, w.low[s].w};
    const uint32_t highs[4] = {w.high[s].x, w.high[s].y, w.high[s].z, w.high[s].w};
    const uint32_t bs[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                   : "+f"(acc[0]), "+f"(acc[1]), "+f"(acc[2]), "+f"(acc[3])
                   : "r"(few_halves(lows[j])), "r"(few_halves(highs[j])), "r"(few_halves(lows[j] >> 16)), "r"(few_halves(highs[j] >> 16)),
                     "r"(few_halves(bs[j])), "r"(few_halves(bs[j] >> 16)));
  }
  const int row = lane >> 2, column = 2 * (lane & 3);
  *reinterpret_cast<float2*>(&smem->sums[warp][row][column]) = make_float2(acc[0], acc[1]);
  *reinterpret_cast<float2*>(&smem->sums[warp][row + 8][column]) = make_float2(acc[2], acc[3]);
}

// A row's sum for a token, the warps' parts in order.
template <int kTokens>
__device__ __forceinline__ __nv_bfloat16 few_sum(const FewSmem<kTokens>* smem, int row, int token) {
  float sum = smem->sums[0][row][token];
#pragma unroll
  for (int w = 1; w < kFwWarps; ++w) sum = __fadd_rn(sum, smem->sums[w][row][token]);
  return __float2bfloat16_rn(sum);
}

// Scale of a token from the threads' maxima: of all columns, by every thread for itself.
template <int kTokens>
__device__ __forceinline__ void few_maximum(FewSmem<kTokens>* smem, int token, float maximum) {
#pragma unroll
  for (int offset = 16; offset; offset >>= 1) maximum = fmaxf(maximum, __shfl_xor_sync(0xffffffffu, maximum, offset));
  if ((threadIdx.x & 31) == 0) smem->maxima[token][threadIdx.x >> 5] = maximum;
}
template <int kTokens>
__device__ __forceinline__ float few_scale(const FewSmem<kTokens>* smem, int token) {
  float maximum = smem->maxima[token][0];
#pragma unroll
  for (int w = 1; w < kFwWarps; ++w) maximum = fmaxf(maximum, smem->maxima[token][w]);
  return fmaxf(__fdiv_rn(maximum, 448.0f), 1.17549435e-38f);
}

__device__ __forceinline__ uint2 few_encode(const float* v, float inverse) {
  uint32_t pairs[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    pairs[i] = __nv_cvt_float2_to_fp8x2(float2{__fmul_rn(v[2 * i], inverse), __fmul_rn(v[2 * i + 1], inverse)}, __NV_SATFINITE, __NV_E4M3);
  return make_uint2(pairs[0] | pairs[1] << 16, pairs[2] | pairs[3] << 16);
}

__device__ __forceinline__ void few_unpack(const uint4& raw, float* v) {
  const uint32_t words[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(words[i] << 16);
    v[2 * i + 1] = __uint_as_float(words[i] & 0xffff0000u);
  }
}

// Eight rows of the gate and the same of the up projection, and their GeGLU products.  The arithmetic of fp8_quantize_rows_kernel and of
// gelu_quantize_fp8_kernel, bit by bit; CTA 0 also keeps the codes and the scales.
template <int kTokens>
__global__ void __launch_bounds__(kFwThreads, 2)
dense_few_gate_up_kernel(const __nv_bfloat16* __restrict__ input, const uint8_t* __restrict__ weights, uint8_t* __restrict__ codes,
                         float* __restrict__ scales, float gate_w_scale, float up_w_scale, __nv_bfloat16* __restrict__ out,
                         __nv_bfloat16* __restrict__ products, int tokens) {
  constexpr int kSteps = kHidden / (kFwWarps * kFwStepBytes);
  __shared__ FewSmem<kTokens> smem;
  grid_dependency_wait();
  grid_launch_dependents();  // after the wait: whoever starts now may read what came before this kernel
  uint4 raw[kTokens];
#pragma unroll
  for (int t = 0; t < kTokens; ++t)
    raw[t] = t < tokens ? __ldg(reinterpret_cast<const uint4*>(input + static_cast<size_t>(t) * kHidden) + threadIdx.x) : uint4{};
  FewWeights<kSteps> w;
  const uint8_t* const gate_rows = weights + static_cast<size_t>(blockIdx.x) * 8 * kHidden;
  few_fetch(w, gate_rows, gate_rows + static_cast<size_t>(kFwDense) * kHidden);
#pragma unroll
  for (int t = 0; t < kTokens; ++t) {
    float x[8], maximum = 0.0f;
    few_unpack(raw[t], x);
#pragma unroll
    for (int i = 0; i < 8; ++i) maximum = fmaxf(maximum, fabsf(x[i]));
    few_maximum(&smem, t, maximum);
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < kTokens; ++t) {
    float x[8];
    few_unpack(raw[t], x);
    const float scale = few_scale(&smem, t);
    const uint2 code = few_encode(x, __fdiv_rn(1.0f, scale));
    reinterpret_cast<uint2*>(smem.x[t])[threadIdx.x] = code;
    if (blockIdx.x == 0 && t < tokens) {
      reinterpret_cast<uint2*>(codes + static_cast<size_t>(t) * kHidden)[threadIdx.x] = code;
      if (threadIdx.x == 0) scales[t] = scale;
    }
  }
  __syncthreads();
  few_multiply(w, &smem);
  __syncthreads();
  const int token = threadIdx.x >> 3, row = threadIdx.x & 7;
  if (token < tokens) {
    const __nv_bfloat16 gate = few_sum(&smem, row, token), up = few_sum(&smem, row + 8, token);
    const int column = static_cast<int>(blockIdx.x) * 8 + row;
    out[static_cast<size_t>(token) * (2 * kFwDense) + column] = gate;
    out[static_cast<size_t>(token) * (2 * kFwDense) + kFwDense + column] = up;
    const float scale = few_scale(&smem, token);
    const float g = __bfloat162float(__float2bfloat16_rn(__fmul_rn(__bfloat162float(gate), __fmul_rn(scale, gate_w_scale))));
    const float u = __bfloat162float(__float2bfloat16_rn(__fmul_rn(__bfloat162float(up), __fmul_rn(scale, up_w_scale))));
    products[token * kFwDense + column] = __float2bfloat16_rn(__fmul_rn(gv_gelu_tanh(g), u));
  }
}

// The products' quantisation and 16 rows of the down projection, likewise.
template <int kTokens>
__global__ void __launch_bounds__(kFwThreads, 2)
dense_few_down_kernel(const __nv_bfloat16* __restrict__ products, const uint8_t* __restrict__ weights, uint8_t* __restrict__ codes,
                      float* __restrict__ scales, __nv_bfloat16* __restrict__ out, int tokens) {
  constexpr int kSteps = kFwDense / (kFwWarps * kFwStepBytes);
  __shared__ FewSmem<kTokens> smem;
  // The first projection lets this kernel start after its own wait: the weights come from before it.
  FewWeights<kSteps> w;
  const uint8_t* const rows = weights + static_cast<size_t>(blockIdx.x) * kFwRows * kFwDense;
  few_fetch(w, rows, rows + 8 * kFwDense);
  grid_dependency_wait();
  grid_launch_dependents();
  const bool active = threadIdx.x < kFwDense / 8;
  uint4 raw[kTokens];
#pragma unroll
  for (int t = 0; t < kTokens; ++t)
    raw[t] = active && t < tokens ? reinterpret_cast<const uint4*>(products + t * kFwDense)[threadIdx.x] : uint4{};
#pragma unroll
  for (int t = 0; t < kTokens; ++t) {
    float v[8], maximum = 0.0f;
    few_unpack(raw[t], v);
#pragma unroll
    for (int i = 0; i < 8; ++i) maximum = fmaxf(maximum, fabsf(v[i]));
    few_maximum(&smem, t, maximum);
  }
  __syncthreads();
  if (active) {
#pragma unroll
    for (int t = 0; t < kTokens; ++t) {
      float v[8];
      few_unpack(raw[t], v);
      const float scale = few_scale(&smem, t);
      const uint2 code = few_encode(v, __fdiv_rn(1.0f, scale));
      reinterpret_cast<uint2*>(smem.x[t])[threadIdx.x] = code;
      if (blockIdx.x == 0 && t < tokens) {
        reinterpret_cast<uint2*>(codes + static_cast<size_t>(t) * kFwDense)[threadIdx.x] = code;
        if (threadIdx.x == 0) scales[t] = scale;
      }
    }
  }
  __syncthreads();
  few_multiply(w, &smem);
  __syncthreads();
  const int token = threadIdx.x / kFwRows, row = threadIdx.x % kFwRows;
  if (token < tokens) out[static_cast<size_t>(token) * kHidden + blockIdx.x * kFwRows + row] = few_sum(&smem, row, token);
}

static_assert(kDenseFewTokens == 2, "variants");

template <int kTokens>
void launch(const DenseFewOperands& op, int tokens, cudaStream_t stream) {
  launch_chained(dense_few_gate_up_kernel<kTokens>, dim3(kFwDense / 8), dim3(kFwThreads), 0, stream,
                 static_cast<const __nv_bfloat16*>(op.input), op.gate_up_weights, op.act_codes, op.act_scales,
                 op.gate_scale, op.up_scale, static_cast<__nv_bfloat16*>(op.gate_up), static_cast<__nv_bfloat16*>(op.products), tokens);
  const __nv_bfloat16* products = static_cast<const __nv_bfloat16*>(op.products);
  __nv_bfloat16* out = static_cast<__nv_bfloat16*>(op.out);
  if (op.serial_launch)
    dense_few_down_kernel<kTokens><<<kHidden / kFwRows, kFwThreads, 0, stream>>>(products, op.down_weights, op.prod_codes, op.prod_scales, out, tokens);
  else
    launch_chained(dense_few_down_kernel<kTokens>, dim3(kHidden / kFwRows), dim3(kFwThreads), 0, stream, products, op.down_weights,
                   op.prod_codes, op.prod_scales, out, tokens);
}

}  // namespace

void launch_dense_few(const DenseFewOperands& op, int tokens, cudaStream_t stream) {
  if (tokens == 1) launch<1>(op, tokens, stream);
  else launch<2>(op, tokens, stream);
}

}  // namespace gv
