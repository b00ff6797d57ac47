// FP64 square root and division by three, correctly rounded, with few FP64
// instructions: for chains of dependent nodes (the distance sweeps). GB300 takes
// an FP64 instruction from a warp every 63 cycles, whether it depends on the last
// one or not and however many lanes are active, so what counts is how many there
// are: sqrt() has a dozen, this root four; an exact quotient by FMAs three, the
// one on integers none.
#pragma once
#include "esf_fixed.cuh"

namespace esf {

#ifdef __CUDA_ARCH__
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float float_of(unsigned u) { return __uint_as_float(u); }
__device__ __forceinline__ unsigned bits_of(float f) { return __float_as_uint(f); }
#else
inline double fma_rn(double a, double b, double c) { return __builtin_fma(a, b, c); }
inline float fma_rn(float a, float b, float c) { return __builtin_fmaf(a, b, c); }
inline float mul_rn(float a, float b) { return a * b; }
inline float add_rn(float a, float b) { return a + b; }
inline float float_of(unsigned u) {
  float f;
  __builtin_memcpy(&f, &u, 4);
  return f;
}
inline unsigned bits_of(float f) {
  unsigned u;
  __builtin_memcpy(&u, &f, 4);
  return u;
}
#endif
// (double)f of a normal number; below 2^-126, something as small
ESF_HD double widen_normal(float f) {
  const unsigned u = bits_of(f);
  return from_words((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u), u << 29);
}
// the leading 24 bits of x, 2^-126 <= x < 2^128
ESF_HD float leading_float(double x) {
  return float_of(((hi_word(x) - (896u << 20)) << 3) | (lo_word(x) >> 29));
}

// sqrt(x), 2^-60 <= x < 2^60, from y = 1/sqrt(leading_float(x)) with a relative
// error below 2^-20. One Newton step in pairs of floats makes 2^-42 of that; a
// second, by the FP64 residual, a g with |g - sqrt(x)| < 1 ulp; and Tuckerman's
// test decides the last bit (Agarwal, Cooley, Gustavson, Shearer, Slishman and
// Tuckerman, "New scalar and vector elementary functions for the IBM System/370",
// 1986): sqrt(x) lies above the midpoint g + ulp/2 exactly where x > g (g + ulp),
// and below g - ulp/2 exactly where x <= g (g - ulp), ulp being that of the side;
// the residual x - g g is exact, so it is compared with ulp g.
ESF_HD double root_from(double x, float y) {
  const float xh = leading_float(x);
  // the next 23 bits: a float with the exponent of bit 23 and those as fraction,
  // less that power of two
  const unsigned e = ((hi_word(x) >> 20) - 896u - 23u) << 23;
  const float xl = add_rn(float_of(e | ((lo_word(x) & 0x1fffffffu) >> 6)), -float_of(e));
  const float h = mul_rn(0.5f, y), gh = mul_rn(xh, y);
  const float gl = mul_rn(add_rn(fma_rn(-gh, gh, xh), xl), h);
  const double g1 = widen_normal(gh) + widen_normal(gl);
  const double g = fma_rn(fma_rn(-g1, g1, x), widen_normal(h), g1);
  const double d = fma_rn(-g, g, x);
  // ulp g: 2^(e - 52) g, as words of a magnitude; half of it below a power of two
  const unsigned gw = hi_word(g), lw = lo_word(g);
  const unsigned up = gw + (((gw >> 20) - 1023u - 52u) << 20);
  const unsigned down = ((gw & 0xfffffu) | lw) ? up : up - (1u << 20);
  const unsigned dh = hi_word(d) & 0x7fffffffu, dl = lo_word(d);
  const bool neg = hi_word(d) >> 31;
  const bool inc = !neg && (dh > up || (dh == up && dl > lw));
  const bool dec = neg && (dh > down || (dh == down && dl >= lw));
  const unsigned lo = lw + (inc ? 1u : 0u) - (dec ? 1u : 0u);
  const unsigned hi = gw + (inc && lo == 0u ? 1u : 0u) - (dec && lw == 0u ? 1u : 0u);
  return from_words(hi, lo);
}

// t / 3, 2^-1000 <= t: with t's significand N scaled so that N / 3 has 53 bits,
// floor((N + 1) / 3), which is N / 3 to the nearest integer (no ties).
ESF_HD double third_of(double t) {
  const unsigned hi = hi_word(t), lo = lo_word(t);
  const unsigned mh = (hi & 0xfffffu) | 0x100000u;
  const unsigned s = mh >= 0x180000u ? 1u : 2u;  // N >= 2^52 + 2^51: one place, else two
  const unsigned nl = (lo << s) + 1u;            // (even before: no carry)
  const unsigned nh = (mh << s) | (lo >> (32u - s));
  // nh 2^32 + nl by 3, with 2^32 = 3 0x55555555 + 1
  const unsigned qh = nh / 3u, r = nh - 3u * qh;
  const unsigned sum = nl + r;
  const unsigned carry = sum < nl ? 1u : 0u;     // 2^32 more: 0x55555555, and 1 to the remainder
  const unsigned q0 = sum / 3u, r0 = sum - 3u * q0;
  const unsigned ql = r * 0x55555555u + q0 + carry * 0x55555555u + (r0 + carry >= 3u ? 1u : 0u);
  // qh 2^32 + ql in [2^52, 2^53): the hidden bit adds one to the exponent
  return from_words(((hi >> 20) - s - 1u) * (1u << 20) + qh, ql);
}
// t / 2
ESF_HD double half_of(double t) { return from_words(hi_word(t) - (1u << 20), lo_word(t)); }

}  // namespace esf
