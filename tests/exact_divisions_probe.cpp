// Compares the two divisions of gv_exact.h with IEEE division: every significand for the constant
// divisor and for every integer divisor 1..15, a spread of exponents, and every E4M3 scale code; and the
// table form of the tanh GELU with the function itself for every bf16 argument.  Prints the number of differences.
#include <cmath>
#include <cstdint>
#include <cstdio>

#include "../gevva_b200/csrc/gv_exact.h"

static const float reciprocals[GV_RECIPROCAL_FLOATS] = GV_RECIPROCALS_INIT;

static float from_parts(int exponent, uint32_t significand) {
  return gv_bits_to_float((static_cast<uint32_t>(127 + exponent) << 23) | significand);
}

static float scale_value(uint32_t code) {
  return code < 8 ? code * 0.001953125f : std::ldexp(8.0f + (code & 7), static_cast<int>(code >> 3) - 10);
}

static float quotient(float multiplier, uint32_t code) {
  const float value = scale_value(code);
  return value == 0.0f ? 0.0f : multiplier / value;
}

int main() {
  long differences = 0;
  const int exponents[] = {-90, -21, -2, -1, 0, 1, 2, 17, 64, 110};
  for (int exponent : exponents)
    for (uint32_t significand = 0; significand < (1u << 23); ++significand) {
      const float t = from_parts(exponent, significand);
      differences += gv_sixth(t) != t / 6.0f;
    }
  for (uint32_t code = 0; code < 16; ++code)  // divisors 0..15
    for (uint32_t significand = 0; significand < (1u << 23); ++significand) {
      const float m = from_parts(7, significand);
      differences += gv_scale_inverse(m, code, reciprocals) != quotient(m, code);
    }
  for (uint32_t code = 0; code < 128; ++code)
    for (int exponent = -99; exponent < 99; ++exponent)
      for (uint32_t significand = 0; significand < (1u << 23); significand += 8191) {
        const float m = from_parts(exponent, significand);
        differences += gv_scale_inverse_exact(m) && gv_scale_inverse(m, code, reciprocals) != quotient(m, code);
      }
  differences += gv_sixth(0.0f) != 0.0f || !std::isinf(gv_sixth(INFINITY));
  static float table[GV_GELU_FLOATS];
  for (uint32_t i = 0; i < GV_GELU_FLOATS; ++i) table[i] = gv_gelu_entry(i);
  for (uint32_t magnitude = 0; magnitude < 32768; ++magnitude) {
    if (magnitude && magnitude < GV_GELU_FIRST) continue;
    const uint32_t offsets = gv_gelu_offsets(magnitude | (magnitude | 0x8000u) << 16);  // the number and its negative
    for (uint32_t sign = 0; sign < 2; ++sign) {
      const float x = gv_bits_to_float(sign << 31 | magnitude << 16);
      const float direct = gv_gelu_tanh(x), looked_up = x * table[(sign ? offsets >> 16 : offsets & 0xffffu) / 4];
      differences += gv_float_to_bits(direct) != gv_float_to_bits(looked_up) && !(direct != direct && looked_up != looked_up);
    }
  }
  std::printf("%ld\n", differences);
  return 0;
}
