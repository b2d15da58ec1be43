// FP64 quotients and square roots on the integer pipe.
//
// sm_103a issues two FP64 lanes per SM and clock: one FP64 instruction of a
// warp occupies its sub-partition's FP64 unit for 64 cycles, in which some 30
// to 60 integer instructions issue.  The division of the compiler is a chain
// of about eleven FP64 instructions; below it is about sixty integer ones on
// the 53-bit significands, whose result is the correctly rounded quotient
// (IEEE 754 round to nearest even), so the bits are those of `a / b`.
//
// Method: long division with two digits of about 30 and 25 bits.  A
// reciprocal of the divisor's leading 32 bits (single-precision approximation
// and one Newton step in fixed point) gives each digit to within a few units,
// the remainder is exact modulo 2^64, and a last comparison of the remainder
// with the divisor makes the quotient exact.  A quotient of two 53-bit
// numbers is never half way between two 53-bit numbers, and neither is a
// square root, so the rounding needs the next bit alone (Muller et al.,
// Handbook of Floating-Point Arithmetic, 4.5 and 4.7).  Zeros, subnormals,
// infinities, NaN and results near the ends of the exponent range take the
// compiler's operation.
//
// The functions compile for the host too, where the tests compare them with
// the processor's own division and square root.
#pragma once

#include <cmath>
#include <cstring>
#include <stdint.h>

#ifdef __CUDACC__
#define XC_HD __host__ __device__ __forceinline__
#else
#define XC_HD inline
#endif

XC_HD uint64_t xc_bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  std::memcpy(&u, &x, 8);
  return u;
#endif
}
XC_HD double xc_from_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  std::memcpy(&x, &u, 8);
  return x;
#endif
}

#ifndef XC_SEED_ULPS     // the tests move the seeds by the approximations' error
#define XC_SEED_ULPS 0
#endif
// bits of about 1 / f and 1 / sqrt(f) in single precision
XC_HD uint32_t xc_seed_rcp(uint32_t fbits) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fbits)));
  return __float_as_uint(r);
#else
  float f;
  std::memcpy(&f, &fbits, 4);
  f = 1.0f / f;
  uint32_t u;
  std::memcpy(&u, &f, 4);
  return u + (XC_SEED_ULPS);
#endif
}
XC_HD uint32_t xc_seed_rsqrt(uint32_t fbits) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fbits)));
  return __float_as_uint(r);
#else
  float f;
  std::memcpy(&f, &fbits, 4);
  f = 1.0f / std::sqrt(f);
  uint32_t u;
  std::memcpy(&u, &f, 4);
  return u + (XC_SEED_ULPS);
#endif
}
XC_HD uint32_t xc_mulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
XC_HD uint64_t xc_mulwide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }

// single-precision bits, raised to those of 0.5
XC_HD uint32_t xc_not_below_half(uint32_t g) { return g < 0x3f000000u ? 0x3f000000u : g; }

// a / b, correctly rounded
XC_HD double xc_div(double a, double b) {
  const uint64_t ua = xc_bits(a), ub = xc_bits(b);
  const uint32_t ha = (uint32_t)(ua >> 32), hb = (uint32_t)(ub >> 32);
  const int ea = (int)((ha >> 20) & 0x7ffu), eb = (int)((hb >> 20) & 0x7ffu);
  const int e0 = ea - eb + 1023;
  // both operands normal, the quotient's exponent well inside the range
  if ((unsigned)(ea - 1) < 2046u && (unsigned)(eb - 1) < 2046u && (unsigned)(e0 - 2) < 2043u) {
    const uint64_t M = (1ull << 52) - 1;
    uint64_t ma = (ua & M) | (1ull << 52);
    const uint64_t mb = (ub & M) | (1ull << 52);
    const int lt = ma < mb ? 1 : 0;
    ma <<= lt;                                               // ma / mb in [1, 2)
    const uint32_t bh = (uint32_t)(mb >> 21);                // leading 32 bits, top bit set
    // r ~ 2^63 / bh from below: 24 bits (six units off: the truncation of bh and the approximation, so
    // that it stays below whatever its rounding), then one Newton step
    const uint32_t g = xc_not_below_half(xc_seed_rcp(0x3f800000u | ((bh >> 8) & 0x7fffffu)) - 6u);
    const uint32_t r0 = ((g & 0x7fffffu) | 0x800000u) << 8;
    const uint64_t err = (1ull << 63) - xc_mulwide(bh, r0);  // in [0, 2^44)
    const uint32_t r = r0 + (xc_mulhi(r0, (uint32_t)(err >> 12)) >> 19);
    // first digit: ma 2^30 / mb, at most a few units below
    const uint32_t q1 = xc_mulhi((uint32_t)(ma >> 22), r) - 1u;
    const uint32_t mbl = (uint32_t)mb, mbh = (uint32_t)(mb >> 32);
    const uint64_t rem1 = (ma << 30) - (xc_mulwide(q1, mbl) + ((uint64_t)(q1 * mbh) << 32));   // in [0, 8 mb)
    // second digit: rem1 2^23 / mb to within one unit
    const uint32_t q2 = xc_mulhi((uint32_t)(rem1 >> 24), r) >> 5;
    const int64_t rem2 = (int64_t)((rem1 << 23) - (xc_mulwide(q2, mbl) + ((uint64_t)(q2 * mbh) << 32)));
    uint64_t q = ((uint64_t)q1 << 23) + q2;                  // floor(ma 2^53 / mb) to within one
    q = rem2 < 0 ? q - 1 : (rem2 >= (int64_t)mb ? q + 1 : q);
    const uint64_t mant = (q + 1) >> 1;                      // with its leading bit, which adds one to the exponent
    return xc_from_bits(((uint64_t)((ha ^ hb) & 0x80000000u) << 32) + ((uint64_t)(uint32_t)(e0 - lt - 1) << 52) + mant);
  }
  return a / b;
}

// sqrt(a), correctly rounded
XC_HD double xc_sqrt(double a) {
  const uint64_t ua = xc_bits(a);
  const uint32_t ha = (uint32_t)(ua >> 32);
  if (ha - 0x00100000u < 0x7fe00000u) {                      // positive, normal, finite
    const int e = (int)(ha >> 20);                           // biased exponent
    const int odd = (e & 1) ^ 1;                             // 1: significand taken in [2, 4)
    const uint64_t mm = ((ua & ((1ull << 52) - 1)) | (1ull << 52)) << odd;   // [2^52, 2^54)
    const uint32_t fh = (uint32_t)(mm >> 22);                // f 2^30, f in [1, 4)
    const uint32_t g = xc_not_below_half(
        xc_seed_rsqrt(((uint32_t)(127 + odd) << 23) | ((ha << 3) & 0x7ffff8u) | ((uint32_t)ua >> 29)) - 8u);
    const uint32_t y0 = ((g & 0x7fffffu) | 0x800000u) << 8;  // 2^32 / sqrt(f), from below
    const uint64_t p = xc_mulwide(fh, xc_mulhi(y0, y0));
    const uint64_t err = (1ull << 62) - p;                   // 1 - f y^2, in 2^62, >= 0
    const uint32_t y = y0 + (xc_mulhi(y0, (uint32_t)(err >> 12)) >> 19);
    const uint32_t s1 = xc_mulhi(fh, y) - 1u;                // sqrt(f) 2^30, at most a few units below
    const uint64_t R1 = (mm << 8) - xc_mulwide(s1, s1);
    const uint32_t s2 = xc_mulhi((uint32_t)(R1 >> 4), y) >> 4;
    uint64_t S = ((uint64_t)s1 << 23) + s2;                  // floor(sqrt(mm 2^54)) to within one
    const int64_t rem = (int64_t)((mm << 54) - S * S);
    S = rem < 0 ? S - 1 : (rem > (int64_t)(2 * S) ? S + 1 : S);
    const uint64_t mant = (S + 1) >> 1;
    return xc_from_bits(((uint64_t)(uint32_t)((e + 1023 - odd) >> 1) << 52) + (mant - (1ull << 52)));
  }
  return std::sqrt(a);
}
