// sin of binary32 arguments as the colour's noise uses it: se_sin, defined by its binary64
// operations, and se_sin_fast, the same bits from integer arithmetic.
#pragma once
#include <cstdint>

namespace se::rt {

// sin of a binary32 argument: evaluated in binary64 and rounded once to binary32.
// Argument reduction by Cody and Waite's method (W. J. Cody, W. Waite, Software Manual for
// the Elementary Functions, 1980): k = the nearest integer to x * 2/pi, r = x - k * pi/2
// with pi/2 split into three 21-bit parts (k * part is exact for |k| < 2^32) and a
// binary64 tail, so r carries about 2^-100 absolute error for |x| < 2^30.  Then the Taylor
// series of sin (to r^17) or cos (to r^18) on |r| <= pi/4 (truncation below 1e-19),
// chosen and signed by k mod 4.  The result is the correctly rounded sinf(x) except when
// the binary64 value lies within about 1e-16 (relative) of a rounding boundary; it is
// within 1 ulp of sin(x), inside CUDA's documented 2-ulp bound for sinf.  Every operation
// is an explicit round-to-nearest binary64 intrinsic (no contraction), so the CPU oracle's
// restatement gives the same bits.  |x| < 2^-12 gives x (the correctly rounded value);
// |x| >= 2^52 (never met: the noise's arguments stay below 2^30) gives x - x (NaN for
// infinities and NaN, else 0).
__device__ __forceinline__ float se_sin(float xf) {
  const double x = (double)xf;
  if (!(fabs(x) < 0x1p52)) return (float)__dsub_rn(x, x);
  if (fabs(x) < 0x1p-12) return xf;  // sin(x) rounds to x (keeps the sign of zero)
  const double k = floor(__dadd_rn(__dmul_rn(x, 0x1.45f306dc9c883p-1), 0.5));
  double r = __dsub_rn(x, __dmul_rn(k, 0x1.921fb0p+0));
  r = __dsub_rn(r, __dmul_rn(k, 0x1.5110bp-22));
  r = __dsub_rn(r, __dmul_rn(k, 0x1.18469p-44));
  r = __dsub_rn(r, __dmul_rn(k, 0x1.13198a2e03707p-65));
  const double r2 = __dmul_rn(r, r);
  // Taylor coefficients (-1)^n / (2n+1)! and (-1)^n / (2n)!, rounded to binary64
  double ps = 0x1.952c77030ad4ap-49;                       // 1/17!
  ps = __dadd_rn(__dmul_rn(ps, r2), -0x1.ae7f3e733b81fp-41);  // -1/15!
  ps = __dadd_rn(__dmul_rn(ps, r2), 0x1.6124613a86d09p-33);   // 1/13!
  ps = __dadd_rn(__dmul_rn(ps, r2), -0x1.ae64567f544e4p-26);  // -1/11!
  ps = __dadd_rn(__dmul_rn(ps, r2), 0x1.71de3a556c734p-19);   // 1/9!
  ps = __dadd_rn(__dmul_rn(ps, r2), -0x1.a01a01a01a01ap-13);  // -1/7!
  ps = __dadd_rn(__dmul_rn(ps, r2), 0x1.1111111111111p-7);    // 1/5!
  ps = __dadd_rn(__dmul_rn(ps, r2), -0x1.5555555555555p-3);   // -1/3!
  const double sn = __dadd_rn(r, __dmul_rn(__dmul_rn(r, r2), ps));
  double pc = -0x1.6827863b97d97p-53;                      // -1/18!
  pc = __dadd_rn(__dmul_rn(pc, r2), 0x1.ae7f3e733b81fp-45);   // 1/16!
  pc = __dadd_rn(__dmul_rn(pc, r2), -0x1.93974a8c07c9dp-37);  // -1/14!
  pc = __dadd_rn(__dmul_rn(pc, r2), 0x1.1eed8eff8d898p-29);   // 1/12!
  pc = __dadd_rn(__dmul_rn(pc, r2), -0x1.27e4fb7789f5cp-22);  // -1/10!
  pc = __dadd_rn(__dmul_rn(pc, r2), 0x1.a01a01a01a01ap-16);   // 1/8!
  pc = __dadd_rn(__dmul_rn(pc, r2), -0x1.6c16c16c16c17p-10);  // -1/6!
  pc = __dadd_rn(__dmul_rn(pc, r2), 0x1.5555555555555p-5);    // 1/4!
  pc = __dadd_rn(__dmul_rn(pc, r2), -0.5);                    // -1/2!
  const double cs = __dadd_rn(1.0, __dmul_rn(r2, pc));
  const double q = __dsub_rn(k, __dmul_rn(4.0, floor(__dmul_rn(k, 0.25))));  // k mod 4, exact
  const double v = q == 0.0 ? sn : q == 1.0 ? cs : q == 2.0 ? -sn : -cs;
  return __double2float_rn(v);
}


// (a * b) >> 64, at most 3 too small (the product of the low halves and two carries are left out).
__device__ __forceinline__ uint64_t mulhi_short(uint64_t a, uint64_t b) {
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
  return (uint64_t)ah * bh + __umulhi(ah, bl) + __umulhi(al, bh);
}

// The bits of se_sin(xf) without binary64 arithmetic, of which this chip does about two
// operations a clock and SM: the sine in 62-bit fixed point with a bound on its error; where all
// values within the bound round to one binary32 number that is the correctly rounded sine, and
// se_sin's too, whose own error (about 2^-52) the bound includes.  Otherwise (about one
// argument in 2^15) and outside 2^6 <= |x| < 2^26: se_sin itself.
//   Reduction (M. Payne, R. Hanek, Radian reduction for trigonometric functions, 1983): x = m 2^e;
// m times the bits of 2/pi that matter, kept to 96 bits, gives x 2/pi mod 4 to 2 units of 2^-62.
// With the nearest whole number taken off, u = |x 2/pi - q| <= 1/2 and v = u^2 <= 1/4, the
// sine is +- u (s0 - s1 v + s2 v^2 - ...) or +- (c0 - c1 v + ...), the Taylor series in pi/2 u.
// Terms 7 to 3 take 32-bit steps, scaled to 2^59 .. 2^36; each is off by under 2 units, so
// the sum from v^3 on by 2 * 2^-36 * 2^-6 = 2^-41; the omitted terms are below 2^-49, the
// 64-bit steps off by some units of 2^-62.  The bound is 2^-40 (2^-40 u + 2^-56 with the factor u).
// tests/test_noise_sine.py compares every binary32 number of the range on the CPU.
__device__ __forceinline__ float se_sin_fast(float xf) {
  const uint32_t bits = __float_as_uint(xf);
  const uint32_t ex = (bits >> 23) & 255u;
  if (ex - 133u >= 20u) return se_sin(xf);  // exponents 6 .. 25
  const uint32_t m = (bits & 0x7fffffu) | 0x800000u;
  const uint32_t sh = 152u - ex;  // 0 .. 19: 2/pi 2^(96 - sh), whose words are
  const uint32_t d0 = __funnelshift_r(0xfc2757d1u, 0x4e441529u, sh), d1 = __funnelshift_r(0x4e441529u, 0xa2f9836eu, sh),
                 d2 = 0xa2f9836eu >> sh;
  const uint64_t mid = (uint64_t)m * d1 + __umulhi(m, d0);
  const uint32_t hi = m * d2 + (uint32_t)(mid >> 32);
  // (hi, mid) = x 2/pi 2^62 mod 2^64: the fraction, signed, times 2^64 and the whole number
  const int64_t g = (int64_t)(((uint64_t)hi << 34) | ((uint64_t)(uint32_t)mid << 2));
  const uint32_t q = (hi + 0x20000000u) >> 30;
  const bool odd = q & 1u;
  const uint64_t a = g < 0 ? 0ull - (uint64_t)g : (uint64_t)g;
  const uint64_t v = mulhi_short(a, a);
  const uint32_t h = (uint32_t)(v >> 31);  // 2 v
  uint32_t p = odd ? 0xdb7127a2u : 0x16fadb9fu;
  p = (odd ? 0xfce9c51cu : 0x1e8f434du) - (__umulhi(p, h) >> 7);
  p = (odd ? 0xd368f951u : 0x1e3074feu) - (__umulhi(p, h) >> 7);
  p = (odd ? 0x787d41a2u : 0x15078348u) - (__umulhi(p, h) >> 7);
  p = (odd ? 0x5574f1f9u : 0x132d2cceu) - (__umulhi(p, h) >> 6);
  const uint64_t pv = (uint64_t)p * (uint32_t)(v >> 32) + __umulhi(p, (uint32_t)v);  // 2^68 p v
  uint64_t r = (odd ? 0x103c1f081b5ac3b3ull : 0x0519af19dd6ab875ull) - (pv >> 6);
  r = (odd ? 0x4ef4f326f9177969ull : 0x295779cc4b7ca57dull) - mulhi_short(r, v);
  r = (odd ? 0x4000000000000000ull : 0x6487ed5110b4611aull) - mulhi_short(r, v);
  uint32_t sign = bits ^ (q << 30);
  uint64_t e = 1ull << 22;
  if (!odd) {
    sign ^= (uint32_t)((uint64_t)g >> 32);
    r = mulhi_short(r, a);
    e = (a >> 42) + 64u;
  }
  const float lo = __ull2float_rn(r - e), up = __ull2float_rn(r + e);
  if (!(lo == up) || r < e) return se_sin(xf);
  return __uint_as_float(__float_as_uint(lo * 0x1p-62f) | (sign & 0x80000000u));
}

}  // namespace se::rt
