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
