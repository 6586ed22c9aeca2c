// The feed-forward steps around the expert path, and the dense FP8 GeGLU MLP that runs
// beside it (30-layer configuration):
//   ff_prepare   dual RMSNorm + router input  (reference: dual_rmsnorm_router_2816_kernel,
//                src/cuda/kernels/normalization.cuh:83-123)
//   fp8 rows     per-row dynamic E4M3 quantisation (quantize_fp8_rows_kernel,
//                src/cuda/kernels/fp8.cuh:2-26)
//   gelu+quant   tanh-GeGLU of the unscaled gate/up outputs, requantised per row
//                (gelu_quantize_fp8_2112_kernel, src/cuda/kernels/fp8.cuh:308-364)
//   ff_finalize  8-route weighted reduce + three RMSNorms + residual + layer scalar
//                (finalize_feedforward_routes_2816_kernel, normalization.cuh:249-377)
// The projections themselves are in dense_gemm_pair.cu and, for the few SMs beside the experts, grouped_gemm.cu in its FP8 form; the whole
// MLP of one or two tokens is dense_few_rows.cu, with the arithmetic of the row kernels here.
// Rows are 2816 wide: 352 threads x 8 columns, 16-byte loads and stores.  Sums of squares
// are folded in one fixed order (thread, shuffle-down tree, warps in order) and the
// reciprocal square root is IEEE, so a CPU can reproduce every bit.
#include "gv_common.cuh"
#include "gv_dense_rows.cuh"
#include "gv_exact.h"
#include "gv_launchers.h"
#include "gv_plan.cuh"

namespace gv {

namespace {

constexpr int kRowThreads = kHidden / 8;  // 352
constexpr int kDenseThreads = 288;        // 264 active threads x 8 columns

__device__ __forceinline__ uint4 pack8(const float* v) {
  uint4 out;
  __nv_bfloat162 p;
  p = __floats2bfloat162_rn(v[0], v[1]); out.x = *reinterpret_cast<uint32_t*>(&p);
  p = __floats2bfloat162_rn(v[2], v[3]); out.y = *reinterpret_cast<uint32_t*>(&p);
  p = __floats2bfloat162_rn(v[4], v[5]); out.z = *reinterpret_cast<uint32_t*>(&p);
  p = __floats2bfloat162_rn(v[6], v[7]); out.w = *reinterpret_cast<uint32_t*>(&p);
  return out;
}

// A thread's sum of squares of its 8 values, then the warp's in lane 0, by a shuffle-down tree (lanes beyond the
// tree keep their own value).
__device__ __forceinline__ float warp_sum_squares(const float* v) {
  float s = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) s = __fmaf_rn(v[i], v[i], s);
#pragma unroll
  for (int offset = 16; offset; offset >>= 1) {
    const float other = __shfl_down_sync(0xffffffffu, s, offset);
    if ((threadIdx.x & 31) + offset < 32) s = __fadd_rn(s, other);
  }
  return s;
}

// The warps' sums folded in order, by every thread for itself: these kernels are chains of latencies (a row a
// block), and one thread that folds for all costs two more barriers and eleven dependent loads.
constexpr int kRowWarps = kRowThreads / 32;  // 11
__device__ __forceinline__ float fold_warps(const float* sums) {
  float total = sums[0];
#pragma unroll
  for (int w = 1; w < kRowWarps; ++w) total = __fadd_rn(total, sums[w]);
  return total;
}

// Inverse root mean square from a row's sum of squares.
__device__ __forceinline__ float inverse_rms(float sum) {
  return gv_rsqrtf(__fadd_rn(__fdiv_rn(sum, static_cast<float>(kHidden)), 1e-6f));
}

__global__ void __launch_bounds__(kRowThreads)
ff_prepare_kernel(const __nv_bfloat16* __restrict__ input, const __nv_bfloat16* __restrict__ dense_weight,
                  const __nv_bfloat16* __restrict__ expert_weight,
                  const __nv_bfloat16* __restrict__ router_scale, __nv_bfloat16* __restrict__ dense_out,
                  __nv_bfloat16* __restrict__ expert_out, __nv_bfloat16* __restrict__ router_out) {
  __shared__ float sums[kRowWarps];
  grid_launch_dependents();
  grid_dependency_wait();
  const size_t base = static_cast<size_t>(blockIdx.x) * kHidden;
  float x[8], dw[8], ew[8], rs[8];
  unpack8(__ldg(reinterpret_cast<const uint4*>(input + base) + threadIdx.x), x);
  unpack8(__ldg(reinterpret_cast<const uint4*>(dense_weight) + threadIdx.x), dw);
  unpack8(__ldg(reinterpret_cast<const uint4*>(expert_weight) + threadIdx.x), ew);
  unpack8(__ldg(reinterpret_cast<const uint4*>(router_scale) + threadIdx.x), rs);
  const float warp_sum = warp_sum_squares(x);
  if ((threadIdx.x & 31) == 0) sums[threadIdx.x >> 5] = warp_sum;
  __syncthreads();
  const float inverse = inverse_rms(fold_warps(sums));
  const float root = gv_rsqrtf(static_cast<float>(kHidden));
  float d[8], e[8], r[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float normalized = __fmul_rn(x[i], inverse);
    d[i] = __fmul_rn(normalized, dw[i]);
    e[i] = __fmul_rn(normalized, ew[i]);
    const float routed = bf16_round(__fmul_rn(bf16_round(normalized), rs[i]));
    r[i] = __fmul_rn(routed, root);
  }
  reinterpret_cast<uint4*>(dense_out + base)[threadIdx.x] = pack8(d);
  reinterpret_cast<uint4*>(expert_out + base)[threadIdx.x] = pack8(e);
  reinterpret_cast<uint4*>(router_out + base)[threadIdx.x] = pack8(r);
}

__device__ __forceinline__ float low_half(uint32_t pair) { return __uint_as_float(pair << 16); }
__device__ __forceinline__ float high_half(uint32_t pair) { return __uint_as_float(pair & 0xffff0000u); }
__device__ __forceinline__ uint32_t bf16_pair(float low, float high) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(low, high);
  return *reinterpret_cast<const uint32_t*>(&p);
}

__device__ __forceinline__ unsigned long long two_of(uint32_t pair) { return two(low_half(pair), high_half(pair)); }
__device__ __forceinline__ uint32_t round2(unsigned long long v) {
  float low, high;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(low), "=f"(high) : "l"(v));
  return bf16_pair(low, high);
}

template <int kWarps>
__device__ __forceinline__ float block_max(float v, float* scratch) {
#pragma unroll
  for (int offset = 16; offset; offset >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, offset));
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  float total = scratch[0];
#pragma unroll
  for (int w = 1; w < kWarps; ++w) total = fmaxf(total, scratch[w]);
  return total;
}

// Larger of a and |b|, two bf16 numbers a word.  A NaN counts as nothing, as in fmaxf.
__device__ __forceinline__ uint32_t abs_max_pair(uint32_t a, uint32_t b) {
  const uint32_t magnitude = b & 0x7fff7fffu;
  const __nv_bfloat162 m = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&magnitude));
  return *reinterpret_cast<const uint32_t*>(&m);
}

// weights_ahead: the kernel behind this asks for its weights without waiting for it, so it may start only once what came before this has
// completed (the weights may come from there).
__global__ void __launch_bounds__(kRowThreads)
fp8_quantize_rows_kernel(const __nv_bfloat16* __restrict__ input, uint8_t* __restrict__ out,
                         float* __restrict__ scales, int rows, bool weights_ahead, RoutePlan plan) {
  __shared__ float scratch[kRowWarps];
  __shared__ int scan_scratch[16];
  if (!weights_ahead) grid_launch_dependents();
  grid_dependency_wait();
  if (weights_ahead) grid_launch_dependents();
  // the projections are grouped GEMMs with a single "expert" that owns every row: their plan
  if (blockIdx.x == 0 && threadIdx.x < kExperts) publish_groups(threadIdx.x == 0 ? rows : 0, rows, plan, scan_scratch);
  const size_t base = static_cast<size_t>(blockIdx.x) * kHidden;
  float x[8];
  unpack8(__ldg(reinterpret_cast<const uint4*>(input + base) + threadIdx.x), x);
  float maximum = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) maximum = fmaxf(maximum, fabsf(x[i]));
  maximum = block_max<kRowWarps>(maximum, scratch);
  const float scale = e4m3_row_scale(maximum);
  if (threadIdx.x == 0) scales[blockIdx.x] = scale;
  const float inverse = __fdiv_rn(1.0f, scale);
  reinterpret_cast<uint2*>(out + base)[threadIdx.x] = encode_e4m3x8(x, inverse);
}

// The same for large batches, a warp a row: the row is held in registers, so that eleven loads of a lane are in flight at once,
// no warp waits for another and a row's scale is computed by one warp, not eleven.  Dense MLP alone, us, a block and a warp a row: 640 tokens
// 29.7 and 29.8, 1024 33.0 and 32.8, 2048 53.5 and 52.7, 4096 92.7 and 91.4; two whole layers in a graph 1024 302 and 305, 2048 440 and 438 (both within
// the spread), 4096 755 and 737.
constexpr int kWarpRows = 8;                    // rows (warps) of a CTA
constexpr int kLaneVectors = kRowThreads / 32;  // 11 vectors of 8 columns a lane

__global__ void __launch_bounds__(kWarpRows * 32)
fp8_quantize_warp_rows_kernel(const __nv_bfloat16* __restrict__ input, uint8_t* __restrict__ out,
                              float* __restrict__ scales, int rows, bool weights_ahead, RoutePlan plan) {
  __shared__ int scan_scratch[16];
  if (!weights_ahead) grid_launch_dependents();
  grid_dependency_wait();
  if (weights_ahead) grid_launch_dependents();
  if (blockIdx.x == 0 && threadIdx.x < kExperts) publish_groups(threadIdx.x == 0 ? rows : 0, rows, plan, scan_scratch);
  const int row = blockIdx.x * kWarpRows + threadIdx.x / 32, lane = threadIdx.x & 31;
  if (row >= rows) return;
  const size_t base = static_cast<size_t>(row) * kHidden;
  uint4 raw[kLaneVectors];
#pragma unroll
  for (int j = 0; j < kLaneVectors; ++j) raw[j] = __ldg(reinterpret_cast<const uint4*>(input + base) + 32 * j + lane);
  uint32_t maxima = 0;
#pragma unroll
  for (int j = 0; j < kLaneVectors; ++j)
    maxima = abs_max_pair(abs_max_pair(abs_max_pair(abs_max_pair(maxima, raw[j].x), raw[j].y), raw[j].z), raw[j].w);
  float maximum = fmaxf(__uint_as_float(maxima << 16), __uint_as_float(maxima & 0xffff0000u));
#pragma unroll
  for (int offset = 16; offset; offset >>= 1) maximum = fmaxf(maximum, __shfl_xor_sync(0xffffffffu, maximum, offset));
  const float scale = e4m3_row_scale(maximum);
  if (lane == 0) scales[row] = scale;
  const float inverse = __fdiv_rn(1.0f, scale);
#pragma unroll
  for (int j = 0; j < kLaneVectors; ++j) {
    float x[8];
    unpack8(raw[j], x);
    reinterpret_cast<uint2*>(out + base)[32 * j + lane] = encode_e4m3x8(x, inverse);
  }
}

__global__ void __launch_bounds__(kDenseThreads)
gelu_quantize_fp8_kernel(const __nv_bfloat16* __restrict__ gate_up,
                         const float* __restrict__ activation_scales, float gate_w_scale,
                         float up_w_scale, uint8_t* __restrict__ out, float* __restrict__ scales) {
  __shared__ float scratch[kDenseThreads / 32];
  grid_dependency_wait();
  grid_launch_dependents();  // the second projection's CTAs take the SMs that the first one leaves, not others
  const int row = blockIdx.x;
  const bool active = threadIdx.x < kDense / 8;
  const float gate_scale = __fmul_rn(activation_scales[row], gate_w_scale);
  const float up_scale = __fmul_rn(activation_scales[row], up_w_scale);
  float value[8];
  float maximum = 0.0f;
  if (active) {
    float g[8], u[8];
    const uint4* src = reinterpret_cast<const uint4*>(gate_up + static_cast<size_t>(row) * 2 * kDense);
    unpack8(__ldg(src + threadIdx.x), g);
    unpack8(__ldg(src + kDense / 8 + threadIdx.x), u);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      value[i] = geglu_tanh(g[i], u[i], gate_scale, up_scale);
      maximum = fmaxf(maximum, fabsf(value[i]));
    }
  }
  maximum = block_max<kDenseThreads / 32>(maximum, scratch);
  const float scale = e4m3_row_scale(maximum);
  if (threadIdx.x == 0) scales[row] = scale;
  const float inverse = __fdiv_rn(1.0f, scale);
  if (active)
    reinterpret_cast<uint2*>(out + static_cast<size_t>(row) * kDense)[threadIdx.x] =
        encode_e4m3x8(value, inverse);
}

// The same for large batches, a warp a row, the row's results held in registers as bf16 pairs; a warp asks for its next columns
// before it works on the ones it has.  The form above is bound by its instructions: the
// exponentials and divisions, and the scale and the folding of maxima in each of nine warps.  Here the tanh factor of a gate is looked up in shared memory,
// the indices and the maxima are made two to a word, and a row's scale is computed once.  Dense MLP alone, us, that form and
// this one: 301 tokens 25.3 and 26.6, 512 26.5 and 26.9, 640 29.6 and 27.9, 1024 32.9 and 31.7, 2048 53.5 and 48.5, 4096 92.7 and 82.4
// (the look-up alone, with a block a row: 53.7 and 91.2).
constexpr int kGeluVectors = (kDense / 8 + 31) / 32;  // 9 vectors of 8 columns a lane, the last in a quarter of the lanes
constexpr int kGeluAtOnce = 3;                        // asked for together
constexpr int kGeluCtas = 2;                          // of an SM
static_assert(kGeluVectors % kGeluAtOnce == 0, "columns in whole steps");

// Gates too small for the table (and, for simplicity, zeros).
__device__ __noinline__ uint32_t gelu_pair_direct(uint32_t gates, uint32_t ups) {
  return bf16_pair(__fmul_rn(gv_gelu_tanh(low_half(gates)), low_half(ups)), __fmul_rn(gv_gelu_tanh(high_half(gates)), high_half(ups)));
}

__device__ __forceinline__ uint32_t scaled_pair(uint32_t pair, float scale) {
  return bf16_pair(__fmul_rn(low_half(pair), scale), __fmul_rn(high_half(pair), scale));
}

__global__ void __launch_bounds__(kWarpRows * 32, kGeluCtas)
gelu_table_quantize_fp8_kernel(const __nv_bfloat16* __restrict__ gate_up, const float* __restrict__ activation_scales,
                               float gate_w_scale, float up_w_scale, const float* __restrict__ gelu_table,
                               uint8_t* __restrict__ out, float* __restrict__ scales, int rows) {
  __shared__ __align__(16) float table[GV_GELU_FLOATS];
  for (int i = threadIdx.x; i < static_cast<int>(GV_GELU_FLOATS / 4); i += kWarpRows * 32)
    reinterpret_cast<float4*>(table)[i] = __ldg(reinterpret_cast<const float4*>(gelu_table) + i);
  __syncthreads();
  grid_dependency_wait();
  grid_launch_dependents();
  const int lane = threadIdx.x & 31;
  for (int row = blockIdx.x * kWarpRows + threadIdx.x / 32; row < rows; row += gridDim.x * kWarpRows) {
    const float activation_scale = __ldg(activation_scales + row);
    const float gate_scale = __fmul_rn(activation_scale, gate_w_scale);
    const float up_scale = __fmul_rn(activation_scale, up_w_scale);
    const uint4* src = reinterpret_cast<const uint4*>(gate_up + static_cast<size_t>(row) * 2 * kDense) + lane;
    uint4 gates[2][kGeluAtOnce], ups[2][kGeluAtOnce];
    auto fetch = [&](int first, int side) {
#pragma unroll
      for (int j = 0; j < kGeluAtOnce; ++j) {
        const int column = 32 * (first + j);
        const bool there = column + lane < kDense / 8;
        gates[side][j] = there ? __ldg(src + column) : uint4{};
        ups[side][j] = there ? __ldg(src + kDense / 8 + column) : uint4{};
      }
    };
    uint32_t value[kGeluVectors][4];
    uint32_t maxima = 0;
    fetch(0, 0);
#pragma unroll
    for (int step = 0; step < kGeluVectors / kGeluAtOnce; ++step) {
      if (step + 1 < kGeluVectors / kGeluAtOnce) fetch((step + 1) * kGeluAtOnce, (step + 1) & 1);
#pragma unroll
      for (int j = 0; j < kGeluAtOnce; ++j) {
        uint32_t g[4] = {gates[step & 1][j].x, gates[step & 1][j].y, gates[step & 1][j].z, gates[step & 1][j].w};
        uint32_t u[4] = {ups[step & 1][j].x, ups[step & 1][j].y, ups[step & 1][j].z, ups[step & 1][j].w};
        uint32_t smallest = 0xffffffffu;
        uint32_t* v = value[step * kGeluAtOnce + j];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          g[i] = scaled_pair(g[i], gate_scale);
          u[i] = scaled_pair(u[i], up_scale);
          smallest = __vminu2(smallest, g[i] & 0x7fff7fffu);
          const uint32_t offsets = gv_gelu_offsets(g[i]);
          const float low = *reinterpret_cast<const float*>(reinterpret_cast<const char*>(table) + (offsets & 0xffffu));
          const float high = *reinterpret_cast<const float*>(reinterpret_cast<const char*>(table) + (offsets >> 16));
          v[i] = bf16_pair(__fmul_rn(__fmul_rn(low_half(g[i]), low), low_half(u[i])),
                           __fmul_rn(__fmul_rn(high_half(g[i]), high), high_half(u[i])));
        }
        const bool there = 32 * (step * kGeluAtOnce + j) + lane < kDense / 8;
        if (there && ((smallest & 0xffffu) < GV_GELU_FIRST || (smallest >> 16) < GV_GELU_FIRST)) {
#pragma unroll
          for (int i = 0; i < 4; ++i) v[i] = gelu_pair_direct(g[i], u[i]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) maxima = abs_max_pair(maxima, v[i]);
      }
    }
    float maximum = fmaxf(__uint_as_float(maxima << 16), __uint_as_float(maxima & 0xffff0000u));
#pragma unroll
    for (int offset = 16; offset; offset >>= 1) maximum = fmaxf(maximum, __shfl_xor_sync(0xffffffffu, maximum, offset));
    const float scale = e4m3_row_scale(maximum);
    if (lane == 0) scales[row] = scale;
    const float inverse = __fdiv_rn(1.0f, scale);
    uint2* dst = reinterpret_cast<uint2*>(out + static_cast<size_t>(row) * kDense) + lane;
#pragma unroll
    for (int j = 0; j < kGeluVectors; ++j) {
      float x[8];
      unpack8(uint4{value[j][0], value[j][1], value[j][2], value[j][3]}, x);
      if (32 * j + lane < kDense / 8) dst[32 * j] = encode_e4m3x8(x, inverse);
    }
  }
}

// The routes' weighted sum, three norms and the residual.  Bound by what is in flight: eight routed rows, the dense row and the residual come
// in, 62 KB a token, and a CTA waits at two barriers.  The pairwise arithmetic and asking for the norm weights only once the
// routes are summed leave 56 registers a thread, so that three CTAs share an SM (two before, with everything asked for at the start).  Alone, us:
// 640 tokens 15.3 -> 12.3, 1024 20.5 -> 16.4, 2048 36.9 -> 30.7, 4096 65.5 -> 56.3; four CTAs of 40 registers take as long as three, a warp a row
// 49 at 2048 tokens.  Whole layers: one token 32.2 -> 31.9 a layer, 301 tokens 320 -> 315 (two layers), 640 244 -> 239, 2048 405 -> 393.
__device__ __forceinline__ float warp_sum_squares_of(const uint32_t (&v)[4]) {
  float s = 0.0f;
#pragma unroll
  for (int i = 0; i < 4; ++i) s = __fmaf_rn(high_half(v[i]), high_half(v[i]), __fmaf_rn(low_half(v[i]), low_half(v[i]), s));
#pragma unroll
  for (int offset = 16; offset; offset >>= 1) s = __fadd_rn(s, __shfl_down_sync(0xffffffffu, s, offset));
  return s;  // right in lane 0
}
__device__ __forceinline__ void words(const uint4& v, uint32_t (&out)[4]) {
  out[0] = v.x;
  out[1] = v.y;
  out[2] = v.z;
  out[3] = v.w;
}

// ff_prepare_kernel for more rows than its CTAs that run at once: a CTA keeps the three weights for row after row and asks for the next one under this one's
// arithmetic, which is done on pairs.  The same results.  Alone, us, a block a row and this: 640 rows 5.25 and 4.55, 1024 7.5 and 6.0, 2048 12.8
// and 10.1, 4096 23.5 and 18.3 (two or four CTAs an SM 20.7 and 21.8); feed-forward layers of 2048 tokens 443.1 and 441.9 (two), 3000 276.8 and 275.2, 4096 362.4
// and 358.3.  With a row a CTA it is the slower one (64 rows 2.03 and 2.14; three layers of 301 tokens 314.6 and 316.4).
constexpr int kPrepareCtas = 3;  // of an SM

__global__ void __launch_bounds__(kRowThreads, 3)
ff_prepare_rows_kernel(const __nv_bfloat16* __restrict__ input, const __nv_bfloat16* __restrict__ dense_weight,
                  const __nv_bfloat16* __restrict__ expert_weight,
                  const __nv_bfloat16* __restrict__ router_scale, __nv_bfloat16* __restrict__ dense_out,
                  __nv_bfloat16* __restrict__ expert_out, __nv_bfloat16* __restrict__ router_out, int rows) {
  __shared__ float sums[2][kRowWarps];
  grid_launch_dependents();
  uint32_t dw[4], ew[4], rs[4];
  grid_dependency_wait();
  const uint4* const in = reinterpret_cast<const uint4*>(input) + threadIdx.x;
  int row = blockIdx.x;
  uint4 raw = __ldg(in + static_cast<size_t>(row) * (kHidden / 8));
  words(__ldg(reinterpret_cast<const uint4*>(dense_weight) + threadIdx.x), dw);
  words(__ldg(reinterpret_cast<const uint4*>(expert_weight) + threadIdx.x), ew);
  words(__ldg(reinterpret_cast<const uint4*>(router_scale) + threadIdx.x), rs);
  const float root = gv_rsqrtf(static_cast<float>(kHidden));
#pragma unroll 1
  for (int turn = 0; row < rows; turn ^= 1) {
    uint32_t x[4];
    words(raw, x);
    const int next = row + static_cast<int>(gridDim.x);
    if (next < rows) raw = __ldg(in + static_cast<size_t>(next) * (kHidden / 8));
    const float warp_sum = warp_sum_squares_of(x);
    if ((threadIdx.x & 31) == 0) sums[turn][threadIdx.x >> 5] = warp_sum;
    __syncthreads();  // (the other turn's sums have been read by all: one barrier a row is enough)
    const float inverse = inverse_rms(fold_warps(sums[turn]));
    uint32_t d[4], e[4], r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const unsigned long long normalized = mul2(two_of(x[i]), two(inverse, inverse));
      d[i] = round2(mul2(normalized, two_of(dw[i])));
      e[i] = round2(mul2(normalized, two_of(ew[i])));
      r[i] = round2(mul2(two_of(round2(mul2(two_of(round2(normalized)), two_of(rs[i])))), two(root, root)));
    }
    const size_t at = static_cast<size_t>(row) * (kHidden / 8) + threadIdx.x;
    reinterpret_cast<uint4*>(dense_out)[at] = uint4{d[0], d[1], d[2], d[3]};
    reinterpret_cast<uint4*>(expert_out)[at] = uint4{e[0], e[1], e[2], e[3]};
    reinterpret_cast<uint4*>(router_out)[at] = uint4{r[0], r[1], r[2], r[3]};
    row = next;
  }
}

__global__ void __launch_bounds__(kRowThreads, 3)
ff_finalize_kernel(const __nv_bfloat16* __restrict__ dense, const __nv_bfloat16* __restrict__ dense_weight,
                   const __nv_bfloat16* __restrict__ expert_routes, const float* __restrict__ route_weights,
                   const int* __restrict__ inverse_routes, const __nv_bfloat16* __restrict__ expert_weight,
                   const __nv_bfloat16* __restrict__ combined_weight, const __nv_bfloat16* __restrict__ residual,
                   const __nv_bfloat16* __restrict__ layer_scalar, __nv_bfloat16* __restrict__ output,
                   const float* __restrict__ dense_activation_scales, const float* __restrict__ dense_projection_scale) {
  __shared__ float dense_sums[kRowWarps], expert_sums[kRowWarps], combined_sums[kRowWarps];
  grid_launch_dependents();
  grid_dependency_wait();
  const int row = blockIdx.x;
  const size_t base = static_cast<size_t>(row) * kHidden;
  uint4 routes[kTopK];
#pragma unroll
  for (int k = 0; k < kTopK; ++k) {
    const int index = row * kTopK + k;
    const int source = inverse_routes ? inverse_routes[index] : index;
    routes[k] = __ldg(reinterpret_cast<const uint4*>(expert_routes + static_cast<size_t>(source) * kHidden) + threadIdx.x);
  }
  uint32_t d[4], e[4], w[4], v[4];
  words(__ldg(reinterpret_cast<const uint4*>(dense + base) + threadIdx.x), d);
  const float scale = dense_activation_scales ? __fmul_rn(dense_activation_scales[row], dense_projection_scale[0]) : 1.0f;
  if (dense_activation_scales) {
#pragma unroll
    for (int i = 0; i < 4; ++i) d[i] = round2(mul2(two_of(d[i]), two(scale, scale)));
  }
  const float dense_sum = warp_sum_squares_of(d);
  unsigned long long sum[4] = {};
#pragma unroll
  for (int k = 0; k < kTopK; ++k) {
    const float weight = route_weights[row * kTopK + k];
    words(routes[k], v);
#pragma unroll
    for (int i = 0; i < 4; ++i) sum[i] = fma2(two_of(v[i]), two(weight, weight), sum[i]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) e[i] = round2(sum[i]);
  const uint4 dense_weight_raw = __ldg(reinterpret_cast<const uint4*>(dense_weight) + threadIdx.x);
  const uint4 expert_weight_raw = __ldg(reinterpret_cast<const uint4*>(expert_weight) + threadIdx.x);
  const uint4 combined_weight_raw = __ldg(reinterpret_cast<const uint4*>(combined_weight) + threadIdx.x);
  const uint4 residual_raw = __ldg(reinterpret_cast<const uint4*>(residual + base) + threadIdx.x);
  const float scalar = __bfloat162float(*layer_scalar);
  const float expert_sum = warp_sum_squares_of(e);
  if ((threadIdx.x & 31) == 0) {
    dense_sums[threadIdx.x >> 5] = dense_sum;
    expert_sums[threadIdx.x >> 5] = expert_sum;
  }
  __syncthreads();
  const float dense_inverse = inverse_rms(fold_warps(dense_sums));
  const float expert_inverse = inverse_rms(fold_warps(expert_sums));
  words(dense_weight_raw, w);
#pragma unroll
  for (int i = 0; i < 4; ++i) d[i] = round2(mul2(mul2(two_of(d[i]), two(dense_inverse, dense_inverse)), two_of(w[i])));
  words(expert_weight_raw, w);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    e[i] = round2(mul2(mul2(two_of(e[i]), two(expert_inverse, expert_inverse)), two_of(w[i])));
    d[i] = round2(add2(two_of(d[i]), two_of(e[i])));
  }
  const float combined_sum = warp_sum_squares_of(d);
  if ((threadIdx.x & 31) == 0) combined_sums[threadIdx.x >> 5] = combined_sum;
  __syncthreads();
  const float combined_inverse = inverse_rms(fold_warps(combined_sums));
  words(combined_weight_raw, w);
  words(residual_raw, v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t normalized = round2(mul2(mul2(two_of(d[i]), two(combined_inverse, combined_inverse)), two_of(w[i])));
    v[i] = round2(mul2(two_of(round2(add2(two_of(v[i]), two_of(normalized)))), two(scalar, scalar)));
  }
  reinterpret_cast<uint4*>(output + base)[threadIdx.x] = uint4{v[0], v[1], v[2], v[3]};
}

__global__ void fp8_amax_kernel(const float* __restrict__ w, size_t count, unsigned int* amax_bits) {
  float maximum = 0.0f;
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    maximum = fmaxf(maximum, fabsf(w[i]));
  for (int offset = 16; offset; offset >>= 1)
    maximum = fmaxf(maximum, __shfl_xor_sync(0xffffffffu, maximum, offset));
  if ((threadIdx.x & 31) == 0) atomicMax(amax_bits, __float_as_uint(maximum));
}

__global__ void fp8_pack_kernel(const float* __restrict__ w, size_t count, const unsigned int* amax_bits,
                                uint8_t* __restrict__ out, float* __restrict__ scale_out) {
  const float scale = e4m3_row_scale(__uint_as_float(*amax_bits));
  if (blockIdx.x == 0 && threadIdx.x == 0) *scale_out = scale;
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    out[i] = static_cast<uint8_t>(encode_e4m3(__fdiv_rn(w[i], scale)));
}

}  // namespace

void launch_ff_prepare(const void* input, const void* dense_weight, const void* expert_weight,
                       const void* router_scale, void* dense_out, void* expert_out, void* router_out,
                       int rows, cudaStream_t stream) {
  using B = __nv_bfloat16;
  const int ctas = kPrepareCtas * current_sm_count();
  if (ctas > 0 && rows > ctas) {
    launch_chained(ff_prepare_rows_kernel, dim3(ctas), dim3(kRowThreads), 0, stream, static_cast<const B*>(input),
                   static_cast<const B*>(dense_weight), static_cast<const B*>(expert_weight),
                   static_cast<const B*>(router_scale), static_cast<B*>(dense_out), static_cast<B*>(expert_out),
                   static_cast<B*>(router_out), rows);
    return;
  }
  launch_chained(ff_prepare_kernel, dim3(rows), dim3(kRowThreads), 0, stream, static_cast<const B*>(input),
                 static_cast<const B*>(dense_weight), static_cast<const B*>(expert_weight),
                 static_cast<const B*>(router_scale), static_cast<B*>(dense_out), static_cast<B*>(expert_out),
                 static_cast<B*>(router_out));
}

void launch_fp8_quantize_rows(const void* input, uint8_t* out, float* scales, int rows, bool weights_ahead, const RoutePlan& plan,
                              cudaStream_t stream) {
  if (rows >= 1024) {  // figures above the kernel
    launch_chained(fp8_quantize_warp_rows_kernel, dim3((rows + kWarpRows - 1) / kWarpRows), dim3(kWarpRows * 32), 0, stream,
                   static_cast<const __nv_bfloat16*>(input), out, scales, rows, weights_ahead, plan);
    return;
  }
  launch_chained(fp8_quantize_rows_kernel, dim3(rows), dim3(kRowThreads), 0, stream,
                 static_cast<const __nv_bfloat16*>(input), out, scales, rows, weights_ahead, plan);
}

void launch_gelu_quantize_fp8(const void* gate_up, const float* activation_scales, float gate_w_scale,
                              float up_w_scale, const float* gelu_table, uint8_t* out, float* scales, int rows,
                              int sm_count, bool serial_launch, cudaStream_t stream) {
  // Up to four tokens an SM the CTAs of one token all run at once, and a row spread over nine warps is done sooner (figures above the kernel).
  if (!serial_launch && rows > 4 * sm_count) {
    const int all = (rows + kWarpRows - 1) / kWarpRows;
    launch_chained(gelu_table_quantize_fp8_kernel, dim3(all < kGeluCtas * sm_count ? all : kGeluCtas * sm_count),
                   dim3(kWarpRows * 32), 0, stream,
                   static_cast<const __nv_bfloat16*>(gate_up), activation_scales, gate_w_scale, up_w_scale, gelu_table, out, scales,
                   rows);
    return;
  }
  if (serial_launch) {
    gelu_quantize_fp8_kernel<<<rows, kDenseThreads, 0, stream>>>(static_cast<const __nv_bfloat16*>(gate_up), activation_scales,
                                                                 gate_w_scale, up_w_scale, out, scales);
    return;
  }
  launch_chained(gelu_quantize_fp8_kernel, dim3(rows), dim3(kDenseThreads), 0, stream,
                 static_cast<const __nv_bfloat16*>(gate_up), activation_scales, gate_w_scale, up_w_scale, out, scales);
}

void launch_ff_finalize(const void* dense, const void* dense_weight, const void* expert_routes,
                        const float* route_weights, const int* inverse_routes, const void* expert_weight,
                        const void* combined_weight, const void* residual, const void* layer_scalar,
                        void* output, int rows, const float* dense_activation_scales,
                        const float* dense_projection_scale, cudaStream_t stream) {
  using B = __nv_bfloat16;
  launch_chained(ff_finalize_kernel, dim3(rows), dim3(kRowThreads), 0, stream, static_cast<const B*>(dense),
                 static_cast<const B*>(dense_weight), static_cast<const B*>(expert_routes), route_weights, inverse_routes,
                 static_cast<const B*>(expert_weight), static_cast<const B*>(combined_weight),
                 static_cast<const B*>(residual), static_cast<const B*>(layer_scalar), static_cast<B*>(output),
                 dense_activation_scales, dense_projection_scale);
}

void launch_pack_fp8(const float* w, size_t count, uint8_t* out, float* scale_out, cudaStream_t stream) {
  unsigned int* accumulator = nullptr;
  cudaMallocAsync(reinterpret_cast<void**>(&accumulator), sizeof(unsigned int), stream);
  cudaMemsetAsync(accumulator, 0, sizeof(unsigned int), stream);
  fp8_amax_kernel<<<592, 256, 0, stream>>>(w, count, accumulator);
  fp8_pack_kernel<<<592, 256, 0, stream>>>(w, count, accumulator, out, scale_out);
  cudaFreeAsync(accumulator, stream);
}

}  // namespace gv
