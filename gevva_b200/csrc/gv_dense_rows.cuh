// Row arithmetic of the dense FP8 MLP, shared by the row-wise kernels (dense_ff.cu) and the kernels of one or two tokens
// (dense_few_rows.cu), whose codes, scales and products have to be the same bit by bit.
#pragma once

#include "gv_common.cuh"

namespace gv {
namespace {

constexpr int kDense = 2112;

// Eight bf16 values as floats.
__device__ __forceinline__ void unpack8(const uint4& raw, float* out) {
  out[0] = __uint_as_float(raw.x << 16);
  out[1] = __uint_as_float(raw.x & 0xffff0000u);
  out[2] = __uint_as_float(raw.y << 16);
  out[3] = __uint_as_float(raw.y & 0xffff0000u);
  out[4] = __uint_as_float(raw.z << 16);
  out[5] = __uint_as_float(raw.z & 0xffff0000u);
  out[6] = __uint_as_float(raw.w << 16);
  out[7] = __uint_as_float(raw.w & 0xffff0000u);
}

__device__ __forceinline__ float bf16_round(float v) {
  return __bfloat162float(__float2bfloat16_rn(v));
}

// Scale of a row of E4M3 codes, from its largest magnitude.
__device__ __forceinline__ float e4m3_row_scale(float maximum) {
  return fmaxf(__fdiv_rn(maximum, 448.0f), 1.17549435e-38f);
}

// Two values a conversion: half the instructions of one at a time, the same bytes.
__device__ __forceinline__ uint2 encode_e4m3x8(const float* v, float inverse) {
  uint32_t pairs[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    pairs[i] = __nv_cvt_float2_to_fp8x2(float2{__fmul_rn(v[2 * i], inverse), __fmul_rn(v[2 * i + 1], inverse)}, __NV_SATFINITE,
                                        __NV_E4M3);
  return make_uint2(pairs[0] | pairs[1] << 16, pairs[2] | pairs[3] << 16);
}

// GeGLU product of unscaled projections, rounded to bf16 as each of its factors is.
__device__ __forceinline__ float geglu_tanh(float gate, float up, float gate_scale, float up_scale) {
  return bf16_round(__fmul_rn(gv_gelu_tanh(bf16_round(__fmul_rn(gate, gate_scale))), bf16_round(__fmul_rn(up, up_scale))));
}

}  // namespace
}  // namespace gv
