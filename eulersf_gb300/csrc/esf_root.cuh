// Correctly rounded FP64 square root for chains of dependent nodes: 500 cycles of
// latency on GB300 where sqrt() takes 800 (a lone warp, 64 a dependent FP64
// operation).
//
// From an approximate y = 1/sqrt(x) (relative error below 2^-20): g = x y and
// h = y/2 refined together once (Goldschmidt's iteration, with FMAs), then g by
// its residual, after which |g - sqrt(x)| < 1 ulp; and the last bit by Tuckerman's
// test (Agarwal, Cooley, Gustavson, Shearer, Slishman and Tuckerman, "New scalar
// and vector elementary functions for the IBM System/370", 1986): sqrt(x) lies
// above the midpoint g + ulp/2 exactly where x > g (g + ulp), and below g - ulp/2
// exactly where x <= g (g - ulp), ulp being that of the side; the residual
// x - g g is exact, so it is compared with ulp g.
#pragma once
#include "esf_fixed.cuh"

namespace esf {

// sqrt(x) for 2^-100 <= x <= 2^100, y as above
ESF_HD double root_from(double x, double y) {
#ifdef __CUDA_ARCH__
#define ESF_FMA __fma_rn
#else
#define ESF_FMA __builtin_fma
#endif
  const double h0 = from_words(hi_word(y) - (1u << 20), lo_word(y));  // y / 2
  const double g0 = x * y;
  const double r0 = ESF_FMA(-g0, h0, 0.5);
  const double g1 = ESF_FMA(g0, r0, g0), h1 = ESF_FMA(h0, r0, h0);
  const double g = ESF_FMA(ESF_FMA(-g1, g1, x), h1, g1);
  const double d = ESF_FMA(-g, g, x);
#undef ESF_FMA
  // ulp g: 2^(e - 52) g, as words of a magnitude; half of it below a power of two
  const unsigned gh = hi_word(g), gl = lo_word(g);
  const unsigned up = gh + (((gh >> 20) - 1023u - 52u) << 20);
  const unsigned down = ((gh & 0xfffffu) | gl) ? up : up - (1u << 20);
  const unsigned dh = hi_word(d) & 0x7fffffffu, dl = lo_word(d);
  const bool neg = hi_word(d) >> 31;
  const bool inc = !neg && (dh > up || (dh == up && dl > gl));
  const bool dec = neg && (dh > down || (dh == down && dl >= gl));
  const unsigned lo = gl + (inc ? 1u : 0u) - (dec ? 1u : 0u);
  const unsigned hi = gh + (inc && lo == 0u ? 1u : 0u) - (dec && gl == 0u ? 1u : 0u);
  return from_words(hi, lo);
}

}  // namespace esf
