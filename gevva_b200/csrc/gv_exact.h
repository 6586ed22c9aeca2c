// The two divisions of the NVFP4 block quantiser without a divide instruction sequence, correctly
// rounded: quotient by a small constant as an approximation q0 = t*r with r = RN(1/d), its exact
// remainder by one fused multiply-add, and one correction, q = fma(rem, r, q0).  With r correctly rounded
// and no over- or underflow that is RN(t/d) (Markstein, "Computation of elementary functions on the
// IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990, theorem on quotients from a correctly rounded
// reciprocal); tests/test_exact_divisions.py compares both functions with IEEE division over every significand.
// A divide costs the epilogue of the expert GEMM about twenty instructions and a branch, twice per
// sixteen values; these take three and nine.
#pragma once

#include "gv_transcendentals.h"

// {RN(1/k), -k}, k = 0..15; the first entry makes the quotient by zero zero, which is the quantiser's rule.
#define GV_RECIPROCALS_INIT {0.0f, 0.0f, 1.0f, -1.0f, 0.5f, -2.0f, 1.0f / 3.0f, -3.0f, 0.25f, -4.0f, 1.0f / 5.0f, -5.0f, \
                             1.0f / 6.0f, -6.0f, 1.0f / 7.0f, -7.0f, 0.125f, -8.0f, 1.0f / 9.0f, -9.0f, 1.0f / 10.0f, \
                             -10.0f, 1.0f / 11.0f, -11.0f, 1.0f / 12.0f, -12.0f, 1.0f / 13.0f, -13.0f, 1.0f / 14.0f, \
                             -14.0f, 1.0f / 15.0f, -15.0f}
#define GV_RECIPROCAL_FLOATS 32

// t / 6 for t >= 0.  Below 2^-100 the result may be off in its last bit, far under the smallest E4M3
// scale (2^-9) that it is rounded to; an infinite t gives infinity.
GV_HD float gv_sixth(float t) {
  const float r = 1.0f / 6.0f;
  const float q0 = GV_MUL(t, r);
  const float q = GV_FMA(GV_FMA(-6.0f, q0, t), r, q0);
  return q == q ? q : q0;
}

// Whether gv_scale_inverse holds for a multiplier: no step of it leaves the normal range.
GV_HD int gv_scale_inverse_exact(float multiplier) { return multiplier > 1e-30f && multiplier < 1e30f; }

// multiplier / (value of the E4M3 scale `code`), 0 for code 0.  The value is k * 2^(e - 10) with an integer
// k <= 15; the power of two is exact.  `reciprocals` points at the
// table above (a shared-memory copy in kernels: lanes read different entries).
GV_HD float gv_scale_inverse(float multiplier, uint32_t code, const float* reciprocals) {
  const uint32_t exponent = code >> 3;
  const uint32_t k = exponent ? 8u + (code & 7u) : code;
  const float r = reciprocals[2 * k];
  const float q0 = GV_MUL(multiplier, r);
  const float q = GV_FMA(GV_FMA(reciprocals[2 * k + 1], q0, multiplier), r, q0);
  return GV_MUL(q, gv_bits_to_float((137u - (exponent ? exponent : 1u)) << 23));
}

// gv_gelu_tanh(x) as x times a factor from a table, for an x that is a bf16 number of magnitude 2^-14 and up (or zero): one entry for each bf16
// number of [2^-14, 2^3), for each sign; from 2^3 on the factor is the last entry's, 1 or 0 (tanh has long reached its limit).  The entries come
// from the function itself, and its halving is exact wherever it stands in the product, so that both give the same bits
// (tests/test_exact_divisions.py compares every argument).
#define GV_GELU_FIRST (113u << 7)                  // 2^-14 as bf16
#define GV_GELU_LAST ((130u << 7) - 1u)            // the last bf16 number below 2^3
#define GV_GELU_SIGN 4096u                         // where the entries of the negative numbers start
#define GV_GELU_FLOATS (GV_GELU_SIGN + GV_GELU_LAST - GV_GELU_FIRST + 1u)

GV_HD float gv_gelu_entry(uint32_t index) {
  const uint32_t sign = index >= GV_GELU_SIGN ? 1u : 0u;
  uint32_t magnitude = GV_GELU_FIRST + index - sign * GV_GELU_SIGN;
  if (magnitude > GV_GELU_LAST) magnitude = GV_GELU_LAST;  // the gap before the negative numbers
  return GV_MUL(0.5f, gv_gelu_factor(gv_bits_to_float((sign << 31) | (magnitude << 16))));
}

// Two bf16 numbers in a word -> the byte offsets of their factors, in a word.  Magnitudes below the table's get the
// first entry, which is right for zero only.
GV_HD uint32_t gv_gelu_offsets(uint32_t pair) {
  const uint32_t magnitude = pair & 0x7fff7fffu;
#if defined(__CUDA_ARCH__)
  const uint32_t clamped = __vmaxu2(__vminu2(magnitude, GV_GELU_LAST * 0x10001u), GV_GELU_FIRST * 0x10001u);
#else
  uint32_t clamped = 0;
  for (int half = 0; half < 32; half += 16) {
    uint32_t m = (magnitude >> half) & 0xffffu;
    m = m > GV_GELU_LAST ? GV_GELU_LAST : m < GV_GELU_FIRST ? GV_GELU_FIRST : m;
    clamped |= m << half;
  }
#endif
  return ((clamped - GV_GELU_FIRST * 0x10001u) << 2) | ((pair >> 1) & 0x40004000u);
}
