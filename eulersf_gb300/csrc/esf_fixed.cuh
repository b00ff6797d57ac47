// Fixed point for the FP64 pressure stencil. GB300 issues two FP64 operations a
// cycle and SM but 128 32-bit integer ones, so the stencil's sums and products
// (36 FP64 operations a row, five sixths of an FP64 iteration's) run on
// integers.
//
// A number is three limbs of 27 bits, l0 + l1 2^27 + l2 2^54, each in a 32-bit
// register with room for the sum of eight fresh limbs and the sign: an addition
// is three independent adds without carries (three-operand ones where two sums
// meet). 96-bit words with carries measured the same in the products and 2 to 7 %
// slower in the solves.
//
// Scale: values v with |v| < 2^Ev become v 2^(77 - Ev), rounded towards zero to
// an integer below 2^77 in magnitude; node factors 1/m < 2^Em keep their 53-bit
// mantissa and an exponent of their own. Sums of eight values (J^T v), their
// products with 1/m and sums of 24 of those fit the limbs; sums are exact, and
// the products drop what lies below 2^-77 of the largest. A double has 53 bits,
// so a cell's result is nearer to the exact one than FP64 arithmetic's where its
// largest product of a value and a factor lies less than 2^21 below the scales'
// (FIX_SPARE); callers use FP64 for the others (fixed_loses).
//
// Where fixed_ok says no (a bound that is not finite, a negative 1/m, scales
// near the top of the exponent range) callers use FP64, in which NaN and
// infinities travel as they always did.
#pragma once
#include "esf_common.cuh"

namespace esf {

struct Fix {
  int l0, l1, l2;
};
constexpr int FIX_BITS = 27, FIX_MASK = (1 << 27) - 1, FIX_TOP = 77;
ESF_HD Fix operator+(Fix a, Fix b) { return Fix{a.l0 + b.l0, a.l1 + b.l1, a.l2 + b.l2}; }
ESF_HD Fix operator-(Fix a, Fix b) { return Fix{a.l0 - b.l0, a.l1 - b.l1, a.l2 - b.l2}; }

#ifdef __CUDA_ARCH__
__device__ __forceinline__ unsigned shf_r(unsigned lo, unsigned hi, int s) { return __funnelshift_r(lo, hi, s); }
__device__ __forceinline__ unsigned shf_l(unsigned lo, unsigned hi, int s) { return __funnelshift_l(lo, hi, s); }
__device__ __forceinline__ int clz32(unsigned a) { return __clz((int)a); }
__device__ __forceinline__ unsigned hi_word(double x) { return (unsigned)__double2hiint(x); }
__device__ __forceinline__ unsigned lo_word(double x) { return (unsigned)__double2loint(x); }
__device__ __forceinline__ double from_words(unsigned hi, unsigned lo) { return __hiloint2double((int)hi, (int)lo); }
#else
inline unsigned shf_r(unsigned lo, unsigned hi, int s) {
  return (unsigned)((((unsigned long long)hi << 32) | lo) >> (s & 31));
}
inline unsigned shf_l(unsigned lo, unsigned hi, int s) {
  return (unsigned)(((((unsigned long long)hi << 32) | lo) << (s & 31)) >> 32);
}
inline int clz32(unsigned a) { return a ? __builtin_clz(a) : 32; }
inline unsigned hi_word(double x) {
  unsigned long long u;
  __builtin_memcpy(&u, &x, 8);
  return (unsigned)(u >> 32);
}
inline unsigned lo_word(double x) {
  unsigned long long u;
  __builtin_memcpy(&u, &x, 8);
  return (unsigned)u;
}
inline double from_words(unsigned hi, unsigned lo) {
  unsigned long long u = ((unsigned long long)hi << 32) | lo;
  double x;
  __builtin_memcpy(&x, &u, 8);
  return x;
}
#endif

// Bounds as the high word of a magnitude: |x| < 2^fixed_exp(h) for every x
// whose high word without its sign is at most h.
ESF_HD unsigned fixed_mag(double x) { return hi_word(x) & 0x7fffffffu; }
ESF_HD int fixed_exp(unsigned h) { return (int)((h >> 20) > 1u ? h >> 20 : 1u) - 1022; }
// ... of one value; at least 1 for what is not zero
ESF_HD unsigned fixed_mag1(double x) { return fixed_mag(x) | (lo_word(x) ? 1u : 0u); }
// The scale Ev for values of at most hv and factors of at most hm: the least,
// but so far from the exponent range's ends that neither a value below 2^-1022
// counts nor a result needs one.
ESF_HD int fixed_scale(unsigned hv, unsigned hm) {
  const int e = fixed_exp(hv), low = -850 - fixed_exp(hm);
  return e > -880 && e > low ? e : low > -880 ? low : -880;
}
// whether it had to be above the values' own, or the factors are denormal (their
// last bits may go out)
ESF_HD bool fixed_low(unsigned hv, unsigned hm) {
  return hv && hm && (fixed_scale(hv, hm) != fixed_exp(hv) || hm < 0x00100000u);
}
// whether the scales fit (and no bound is infinite or NaN, no factor negative)
ESF_HD bool fixed_ok(unsigned hv, unsigned hm) {
  return hv < 0x7ff00000u && hm < 0x7ff00000u && fixed_scale(hv, hm) + fixed_exp(hm) < 900;
}

// Where a value or factor stands: |x| < 2^fixed_place(x), at least half of that
// where x is normal; of zero, far below all others.
constexpr int FIX_NOWHERE = -100000;
ESF_HD int fixed_place(double x) { return fixed_mag1(x) ? fixed_exp(fixed_mag(x)) : FIX_NOWHERE; }
// How far below the scales' product, in places, a cell's largest product of a
// value and a factor may lie. A cell's error is some 11 units of 2^(Ev + Em - 77)
// in the mean square. Against the sum of a cell's terms without their signs, by
// how far it lies below (in brackets an FP64 evaluation's): at the scale 8.5e-18
// (3.5e-17), 21 places 1.2e-17 (3.5e-17), 22 places 3.8e-17 (3.6e-17), 24 places
// 1.6e-16, 45 places 6e-10.
constexpr int FIX_SPARE = 21;

// x 2^(77 - Ev) towards zero, for |x| < 2^Ev, Ev at least -880
ESF_HD Fix fixed_from(double x, int Ev) {
  const unsigned hi = hi_word(x), lo = lo_word(x);
  // the mantissa at the top of 96 bits, then down to its place (for x = 0 or
  // denormal the implicit bit is wrong, but goes out below)
  const unsigned mh = (hi & 0xfffffu) | 0x100000u;
  const unsigned xh = shf_l(lo, mh, 11), xl = lo << 11;
  const int t = Ev + 1041 - (int)((hi >> 20) & 0x7ffu);  // at least 19
  // (selects rather than branches: a warp's values differ in magnitude)
  const unsigned h2 = t < 32 ? xh : 0u, h1 = t < 32 ? xl : t < 64 ? xh : 0u,
                 h0 = t < 32 ? 0u : t < 64 ? xl : t < 96 ? xh : 0u;
  const unsigned w0 = shf_r(h0, h1, t), w1 = shf_r(h1, h2, t), w2 = shf_r(h2, 0u, t);
  const int m = (int)hi >> 31;
  const int l0 = (int)(w0 & FIX_MASK), l1 = (int)(shf_r(w0, w1, 27) & FIX_MASK), l2 = (int)shf_r(w1, w2, 22);
  return Fix{(l0 ^ m) - m, (l1 ^ m) - m, (l2 ^ m) - m};
}

// A node's factor 1/m < 2^Em: its mantissa as a 54-bit fraction of two limbs
// (both 0 for a node without an unknown), and how far its exponent lies below Em.
struct NodeFactor {
  int m0, m1;
  int s;
};
ESF_HD NodeFactor factor_from(double m, int Em) {
  const unsigned hi = hi_word(m), lo = lo_word(m);
  const unsigned e = (hi >> 20) & 0x7ffu;
  const unsigned mh = e ? (hi & 0xfffffu) | 0x100000u : hi & 0xfffffu;
  NodeFactor f;
  f.m0 = (int)((lo << 1) & FIX_MASK);
  f.m1 = (int)shf_r(lo, mh, 26);
  f.s = (mh | lo) ? Em + 1022 - (int)(e ? e : 1u) : 0;  // at least 0
  return f;
}
// the limbs of a as 96 bits (two's complement)
ESF_HD void fixed_words(Fix a, unsigned w[3]) {
  a.l1 += a.l0 >> FIX_BITS;
  a.l2 += a.l1 >> FIX_BITS;
  const unsigned l0 = (unsigned)(a.l0 & FIX_MASK), l1 = (unsigned)(a.l1 & FIX_MASK);
  w[0] = l0 | (l1 << 27);
  w[1] = (l1 >> 5) | ((unsigned)a.l2 << 22);
  w[2] = (unsigned)(a.l2 >> 10);
}
// v times the factor, towards minus infinity, at the scale 2^(77 - Ev - Em),
// with fresh limbs
ESF_HD Fix fixed_mul(Fix v, const NodeFactor& f) {
  typedef long long s64;
  const s64 c = ((s64)v.l1 * f.m0 + (s64)v.l0 * f.m1) >> FIX_BITS;
  const s64 t0 = (s64)v.l2 * f.m0 + (s64)v.l1 * f.m1 + c;
  const s64 t1 = (s64)v.l2 * f.m1 + (t0 >> FIX_BITS);
  Fix r{(int)t0 & FIX_MASK, (int)t1 & FIX_MASK, (int)(t1 >> FIX_BITS)};
  if (f.s) {  // (few nodes: those whose 1/m is below half the largest)
    unsigned w[3];
    fixed_words(r, w);
    const unsigned sign = (unsigned)((int)w[2] >> 31);
    int s = f.s < 96 ? f.s : 96;
    while (s >= 32) {
      w[0] = w[1];
      w[1] = w[2];
      w[2] = sign;
      s -= 32;
    }
    const unsigned a = shf_r(w[0], w[1], s), b = shf_r(w[1], w[2], s), c2 = shf_r(w[2], sign, s);
    r = Fix{(int)(a & FIX_MASK), (int)(shf_r(a, b, 27) & FIX_MASK), (int)shf_r(b, c2, 22)};
  }
  return r;
}

// a 2^(E - 77) rounded to the nearest double (ties to even)
ESF_HD double fixed_to(Fix a, int E) {
  typedef unsigned long long u64;
  unsigned w[3];
  fixed_words(a, w);
  const unsigned m = (unsigned)((int)w[2] >> 31);
  // magnitude: complement and add the sign's one
  u64 lo = (((u64)w[1] << 32) | w[0]) ^ (((u64)m << 32) | m);
  unsigned u2 = w[2] ^ m;
  lo += m & 1u;
  u2 += (m & 1u) & (lo == 0);
  unsigned u1 = (unsigned)(lo >> 32), u0 = (unsigned)lo;
  int e = 95 + E - FIX_TOP + 1022;  // biased, less the hidden bit's one, for a top bit at 95
  if (u2 == 0u) {                   // below 2^-19 of the largest
    u2 = u1;
    u1 = u0;
    u0 = 0u;
    e -= 32;
    if (u2 == 0u) {
      if (u1 == 0u) return 0.0;
      u2 = u1;
      u1 = 0u;
      e -= 32;
    }
  }
  const int z = clz32(u2);
  const unsigned H = shf_l(u1, u2, z);
  const unsigned L = shf_l(u0, u1, z) | (u0 << z ? 1u : 0u);
  // 64 bits to 53: half a place less one, plus the last kept bit; a carry out
  // of the mantissa goes into the exponent
  const u64 t = ((u64)H << 32) | L;
  const u64 q = t + (0x3ffu + ((L >> 11) & 1u));
  const unsigned c = q < t ? 1u << 21 : 0u;
  const unsigned hi = ((unsigned)(e - z) << 20) + (unsigned)(q >> 43) + c;
  return from_words(hi | (m & 0x80000000u), (unsigned)(q >> 11));
}

}  // namespace esf
