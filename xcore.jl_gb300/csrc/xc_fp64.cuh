// FP64 quotients, square roots, exponentials and logarithms on the integer pipe.
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
  // a field that is zero where it has not started to move takes this way in every cell
  if (!(ua << 1) && (ub << 1) - 1 < (0x7ffull << 53) - 1) return xc_from_bits((ua ^ ub) & (1ull << 63));
  return a / b;
}

// a b, correctly rounded (a multiplication occupies the FP64 unit for 64 cycles; this is some 40 integer
// instructions: worth it where the FP64 unit is what a kernel waits for).  The 106-bit product of the significands
// is rounded to nearest even; a zero factor gives its zero, and whatever else leaves the normal range takes the FP64
// unit's product, in a call so that it is not issued otherwise.
#ifdef __CUDACC__
__host__ __device__ __noinline__ inline double xc_mul_any(double a, double b) { return a * b; }
#else
inline double xc_mul_any(double a, double b) { return a * b; }
#endif
XC_HD double xc_mul_edge(double a, double b) {
  const uint64_t ua = xc_bits(a), ub = xc_bits(b), inf = 0x7ffull << 53;
  if ((!(ua << 1) && (ub << 1) < inf) || (!(ub << 1) && (ua << 1) < inf)) return xc_from_bits((ua ^ ub) & (1ull << 63));
  return xc_mul_any(a, b);
}
// 63 bits h, the leading one at 62 or 61, and whether any below them is set -> the rounded product; e the biased
// exponent for a leading one at 61
XC_HD uint64_t xc_round63(uint64_t h, uint32_t sticky, int e, uint32_t sign) {
  const int up = (int)(h >> 62);
  h = up ? h : h << 1;
  h |= sticky ? 1u : 0u;
  const uint64_t r = (h + 0x1ff + ((uint32_t)(h >> 10) & 1u)) >> 10;    // with its leading bit, which adds one to the exponent
  return ((uint64_t)(sign & 0x80000000u) << 32) + ((uint64_t)(uint32_t)(e + up - 1) << 52) + r;
}
XC_HD double xc_mul(double a, double b) {
  const uint64_t ua = xc_bits(a), ub = xc_bits(b);
  const uint32_t ha = (uint32_t)(ua >> 32), hb = (uint32_t)(ub >> 32);
  const int ea = (int)((ha >> 20) & 0x7ffu), eb = (int)((hb >> 20) & 0x7ffu), e = ea + eb - 1023;
  if ((unsigned)(ea - 1) < 2046u && (unsigned)(eb - 1) < 2046u && (unsigned)(e - 1) < 2044u) {
    const uint32_t al = (uint32_t)ua, bl = (uint32_t)ub, ah = (ha & 0xfffffu) | 0x100000u, bh = (hb & 0xfffffu) | 0x100000u;
    const uint64_t p = xc_mulwide(al, bl);
    const uint64_t m = xc_mulwide(ah, bl) + (xc_mulwide(al, bh) + (p >> 32));
    const uint64_t h = xc_mulwide(ah, bh) + (m >> 32);
    return xc_from_bits(xc_round63((h << 21) | ((uint32_t)m >> 11), ((uint32_t)m << 21) | (uint32_t)p, e, ha ^ hb));
  }
  return xc_mul_edge(a, b);
}
// a^2 2^-K, K even: the power of two costs nothing here
#ifdef __CUDACC__
__host__ __device__ __noinline__ inline double xc_sqr_any(double a, double scale) { return (a * scale) * (a * scale); }
#else
inline double xc_sqr_any(double a, double scale) { return (a * scale) * (a * scale); }
#endif
template <int K = 0>
XC_HD double xc_sqr(double a) {
  static_assert(K >= 0 && K % 2 == 0 && K < 100, "the scale's root is a power of two");
  const uint64_t ua = xc_bits(a);
  const uint32_t ha = (uint32_t)(ua >> 32);
  const int ea = (int)((ha >> 20) & 0x7ffu), e = 2 * ea - 1023 - K;
  if ((unsigned)(e - 1) < 2044u) {
    const uint32_t al = (uint32_t)ua, ah = (ha & 0xfffffu) | 0x100000u;
    const uint64_t p = xc_mulwide(al, al);
    const uint64_t m = 2 * xc_mulwide(al, ah) + (p >> 32);
    const uint64_t h = xc_mulwide(ah, ah) + (m >> 32);
    return xc_from_bits(xc_round63((h << 21) | ((uint32_t)m >> 11), ((uint32_t)m << 21) | (uint32_t)p, e, 0));
  }
  return ua << 1 ? xc_sqr_any(a, xc_from_bits((uint64_t)(1023 - K / 2) << 52)) : 0.0;
}
// K a for a small odd K: the product of the significand is exact in 64 bits
template <int K>
XC_HD double xc_mul_small(double a) {
  constexpr int L = K < 4 ? 1 : (K < 8 ? 2 : 3);              // K in [2^L, 2^(L+1))
  static_assert(K >= 2 && K < 16, "small factors");
  const uint64_t ua = xc_bits(a);
  const uint32_t ha = (uint32_t)(ua >> 32);
  const int e = (int)((ha >> 20) & 0x7ffu) + L;
  if ((unsigned)(e - L - 1) < 2040u) {
    const uint64_t m = xc_mulwide((uint32_t)ua, K) + ((uint64_t)(((ha & 0xfffffu) | 0x100000u) * K) << 32);
    return xc_from_bits(xc_round63(m << (9 - L), 0, e, ha));
  }
  return xc_mul_edge((double)K, a);
}

// a rounded to a float (a conversion is on the FP64 unit too); results outside its normal range by the compiler's
// conversion, in a call
#ifdef __CUDACC__
__host__ __device__ __noinline__ inline float xc_to_float_any(double a) { return (float)a; }
#else
inline float xc_to_float_any(double a) { return (float)a; }
#endif
XC_HD float xc_from_float_bits(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x;
  std::memcpy(&x, &u, 4);
  return x;
#endif
}
XC_HD float xc_to_float(double a) {
  const uint64_t u = xc_bits(a);
  const uint32_t h = (uint32_t)(u >> 32), sign = h & 0x80000000u;
  const int e = (int)((h >> 20) & 0x7ffu) - 896;
  if ((unsigned)(e - 1) < 253u) {
    const uint64_t m = (u & ((1ull << 52) - 1)) + 0xfffffffull + ((uint32_t)(u >> 29) & 1u);
    return xc_from_float_bits(sign | (((uint32_t)e << 23) + (uint32_t)(m >> 29)));
  }
  return u << 1 ? xc_to_float_any(a) : xc_from_float_bits(sign);
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
  if (!(ua << 1)) return a;
  return std::sqrt(a);
}

// ---------------------------------------------------------------------------
// exact scalings, comparisons
// ---------------------------------------------------------------------------
// x 2^K, K = 1 or -1, -2: the exponent field where x and the result are
// normal.  All cases in integers: an FP64 product on a rare path would be
// predicated, and a predicated FP64 instruction takes its slot all the same.
template <int K>
XC_HD double xc_scale2(double x) {
  static_assert(K == 1 || K == -1 || K == -2, "scale");
  const uint64_t u = xc_bits(x);
  const unsigned e = (unsigned)(u >> 52) & 0x7ffu;
  constexpr unsigned lo = K < 0 ? 1u + (unsigned)-K : 1u, hi = K > 0 ? 2046u - (unsigned)K : 2046u;
  constexpr int up = K > 0 ? K : 0, down = K < 0 ? -K : 0;
  uint64_t r = u + ((uint64_t)up << 52) - ((uint64_t)down << 52);
  if (e - lo > hi - lo) {
    const uint64_t sign = u & (1ull << 63);
    uint64_t n = u ^ sign;
    if (e == 2047u) r = u;                                        // infinity, NaN
    else if (K > 0) r = sign | (e == 0 ? n << up : 0x7ff0000000000000ull);
    else {                                                        // subnormal result: round to even
      if (e == 2) n = ((n & ((1ull << 52) - 1)) | (1ull << 52)) << 1;
      constexpr int k = K < 0 ? down : 1;
      const uint64_t rest = n & ((1ull << k) - 1), half = 1ull << (k - 1);
      n >>= k;
      r = sign | (n + (rest > half || (rest == half && (n & 1))));
    }
  }
  return xc_from_bits(r);
}
XC_HD double xc_half(double x) { return xc_scale2<-1>(x); }

XC_HD bool xc_isnan(double x) { return (xc_bits(x) << 1) > 0xffe0000000000000ull; }
// the order of the reals on the bits of a double that is not NaN (-0 below +0)
XC_HD int64_t xc_order(double x) {
  const int64_t i = (int64_t)xc_bits(x);
  return i ^ (int64_t)((uint64_t)(i >> 63) >> 1);
}
// x > hi ? hi : (x < lo ? lo : x) for 0 < lo < hi; NaN stays
XC_HD double xc_clamp_pos(double x, double lo, double hi) {
  if (xc_isnan(x)) return x;
  const int64_t k = xc_order(x);
  return k > (int64_t)xc_bits(hi) ? hi : (k < (int64_t)xc_bits(lo) ? lo : x);
}
// x >= c for c > 0
XC_HD bool xc_ge_pos(double x, double c) { return (int64_t)xc_bits(x) >= (int64_t)xc_bits(c) && !xc_isnan(x); }
// Julia's max(0.0, x) and, for c > 0, max(x, c): a NaN stays
XC_HD double xc_max0(double x) { return (int64_t)xc_bits(x) < 0 && !xc_isnan(x) ? 0.0 : x; }
XC_HD double xc_max_pos(double x, double c) { return xc_isnan(x) || xc_order(x) > (int64_t)xc_bits(c) ? x : c; }

// ---------------------------------------------------------------------------
// exponential and logarithm: a table of intervals and a short Taylor sum in
// 64-bit fixed point (the classical table-driven scheme, P. T. P. Tang, ACM
// TOMS 15, 1989, in integers), its higher terms in 32 bits.  The tables are
// 2^(j/1024) and log2 of the interval reciprocals from 60-digit arithmetic.
// xc_exp is within 0.502 ulp up to |x| = 1, 0.51 up to 64 and 0.7 up to 708.
// Below 2^-14 it is nearer still: where 1 - exp(-x) of such an x is formed, an
// ulp of exp is 2^14 or more of the difference.
// ---------------------------------------------------------------------------
#ifdef __CUDACC__
#define XC_TABLE static __device__ const
#else
#define XC_TABLE static const
#endif
// 2^(j/1024) 2^63, rounded down
XC_TABLE uint64_t xc_exp2_tab[1024] = {
    0x8000000000000000ull, 0x8016302f17467628ull, 0x802c6436d0e04f50ull, 0x80429c17d77c18edull, 0x8058d7d2d5e5f6b0ull,
    0x806f17687707a7afull, 0x80855ad965e88b83ull, 0x809ba2264dada76aull, 0x80b1ed4fd999ab6cull, 0x80c83c56b50cf77full,
    0x80de8f3b8b85a0afull, 0x80f4e5ff089f763eull, 0x810b40a1d81406d4ull, 0x81219f24a5baa59dull, 0x813801881d886f7bull,
    0x814e67cceb90502cull, 0x8164d1f3bc030773ull, 0x817b3ffd3b2f2e47ull, 0x8191b1ea15813bfdull, 0x81a827baf7838b78ull,
    0x81bea1708dde6055ull, 0x81d51f0b8557ec1cull, 0x81eba08c8ad4536full, 0x820225f44b55b33bull, 0x8218af4373fc25ebull,
    0x822f3c7ab205c89aull, 0x8245cd9ab2cec048ull, 0x825c62a423d13f0cull, 0x8272fb97b2a5894cull, 0x828998760d01faf3ull,
    0x82a0393fe0bb0ca8ull, 0x82b6ddf5dbc35906ull, 0x82cd8698ac2ba1d7ull, 0x82e433290022d54aull, 0x82fae3a785f61332ull,
    0x83119814ec10b242ull, 0x83285071e0fc4546ull, 0x833f0cbf1360a064ull, 0x8355ccfd3203de5aull, 0x836c912cebca65bcull,
    0x8383594eefb6ee36ull, 0x839a2563ecea85cfull, 0x83b0f56c92a49627ull, 0x83c7c9699042e9bdull, 0x83dea15b9541b132ull,
    0x83f57d43513b888full, 0x840c5d2173e97c8bull, 0x842340f6ad230fd0ull, 0x843a28c3acde4046ull, 0x84511489232f8c56ull,
    0x84680447c049f83bull, 0x847ef800347f1347ull, 0x8495efb3303efd2full, 0x84aceb6164186b5bull, 0x84c3eb0b80b8ae2full,
    0x84daeeb236ebb65bull, 0x84f1f656379c1a29ull, 0x850901f833d31acfull, 0x85201198dcb8a9c0ull, 0x85372538e3936dfaull,
    0x854e3cd8f9c8c95dull, 0x85655879d0dcddfcull, 0x857c781c1a729376ull, 0x85939bc0884b9c43ull, 0x85aac367cc487b14ull,
    0x85c1ef1298688825ull, 0x85d91ec19ec9f694ull, 0x85f0527591a9d9c0ull, 0x86078a2f23642a9full, 0x861ec5ef0673cd18ull,
    0x863605b5ed729562ull, 0x864d49848b194d62ull, 0x8664915b923fba03ull, 0x867bdd3bb5dca09cull, 0x86932d25a905cc49ull,
    0x86aa811a1ef01352ull, 0x86c1d919caef5c87ull, 0x86d935256076a4a8ull, 0x86f0953d931803c3ull, 0x8707f9631684b29bull,
    0x871f61969e8d1010ull, 0x8736cdd8df20a67full, 0x874e3e2a8c4e3131ull, 0x8765b28c5a43a1baull, 0x877d2afefd4e256cull,
    0x8794a78329da2ab8ull, 0x87ac28199473669full, 0x87c3acc2f1c4da1cull, 0x87db357ff698d791ull, 0x87f2c25157d90833ull,
    0x880a5337ca8e717bull, 0x8821e83403e17a97ull, 0x88398146b919f1d4ull, 0x88511e709f9f1218ull, 0x8868bfb26cf78850ull,
    0x8880650cd6c978e3ull, 0x88980e8092da8527ull, 0x88afbc0e570fd0d8ull, 0x88c76db6d96e078cull, 0x88df237ad019622cull,
    0x88f6dd5af155ac6bull, 0x890e9b57f3864a3full, 0x89265d728d2e3d5dull, 0x893e23ab74f02ab1ull, 0x8955ee03618e5fdcull,
    0x896dbc7b09ead8b1ull, 0x89858f13250744b1ull, 0x899d65cc6a050c8eull, 0x89b540a7902557a3ull, 0x89cd1fa54ec9117full,
    0x89e502c65d70ef5eull, 0x89fcea0b73bd75afull, 0x8a14d575496efd9aull, 0x8a2cc5049665ba7eull, 0x8a44b8ba12a1bf7full,
    0x8a5cb09676430504ull, 0x8a74ac9a79896e46ull, 0x8a8cacc6d4d4ced3ull, 0x8aa4b11c40a4f018ull, 0x8abcb99b759996eeull,
    0x8ad4c6452c728924ull, 0x8aecd71a1e0f9309ull, 0x8b04ec1b03708cfdull, 0x8b1d054895b560fdull, 0x8b3522a38e1e1031ull,
    0x8b4d442ca60ab87full, 0x8b6569e496fb9a18ull, 0x8b7d93cc1a911d0eull, 0x8b95c1e3ea8bd6e6ull, 0x8badf42cc0cc902bull,
    0x8bc62aa757544a01ull, 0x8bde6554684443bfull, 0x8bf6a434adde0084ull, 0x8c0ee748e2834cceull, 0x8c272e91c0b64413ull,
    0x8c3f7a100319565cull, 0x8c57c9c4646f4dddull, 0x8c701daf9f9b5496ull, 0x8c8875d26fa0f9e9ull, 0x8ca0d22d8fa4383bull,
    0x8cb932c1bae97a95ull, 0x8cd1978facd5a23eull, 0x8cea009820ee0c5full, 0x8d026ddbd2d897a6ull, 0x8d1adf5b7e5ba9e5ull,
    0x8d335517df5e35b7ull, 0x8d4bcf11b1e7c024ull, 0x8d644d49b2206648ull, 0x8d7ccfc09c50e2f7ull, 0x8d9556772ce29468ull,
    0x8dade16e205f81d8ull, 0x8dc670a633726138ull, 0x8ddf042022e69cd5ull, 0x8df79bdcaba85906ull, 0x8e1037dc8ac479d3ull,
    0x8e28d8207d68a8a8ull, 0x8e417ca940e35a01ull, 0x8e5a257792a3d317ull, 0x8e72d28c303a2f94ull, 0x8e8b83e7d7576743ull,
    0x8ea4398b45cd53c0ull, 0x8ebcf377398eb62dull, 0x8ed5b1ac70af3ce9ull, 0x8eee742ba963893full, 0x8f073af5a2013520ull,
    0x8f20060b18fed8dbull, 0x8f38d56cccf410d3ull, 0x8f51a91b7c998338ull, 0x8f6a8117e6c8e5c4ull, 0x8f835d62ca7d0371ull,
    0x8f9c3dfce6d1c23cull, 0x8fb522e6fb0428dbull, 0x8fce0c21c6726481ull, 0x8fe6f9ae089bce98ull, 0x8fffeb8c8120f285ull,
    0x9018e1bdefc39367ull, 0x9031dc431466b1dcull, 0x904adb1caf0e91beull, 0x9063de4b7fe0bfeeull, 0x907ce5d047241815ull,
    0x9095f1abc540ca6bull, 0x90af01debac0617dull, 0x90c81669e84dc7f8ull, 0x90e12f4e0eb54e70ull, 0x90fa4c8beee4b12aull,
    0x91136e2449eb1de7ull, 0x912c9417e0f939b2ull, 0x9145be67756126aaull, 0x915eed13c89689d3ull, 0x9178201d9c2e90e3ull,
    0x91915785b1dff814ull, 0x91aa934ccb830ff4ull, 0x91c3d373ab11c336ull, 0x91dd17fb12a79c87ull, 0x91f660e3c481cc64ull,
    0x920fae2e82ff2ee9ull, 0x9228ffdc10a051acull, 0x924255ed30077996ull, 0x925bb062a3f8a8b4ull, 0x92750f3d2f59a417ull,
    0x928e727d9531f9acull, 0x92a7da2498ab0615ull, 0x92c14632fd0ffa88ull, 0x92dab6a985cde2aeull, 0x92f42b88f673aa7cull,
    0x930da4d212b22415ull, 0x932722859e5c0dabull, 0x9340a4a45d661761ull, 0x935a2b2f13e6e92bull, 0x9373b626861728b3ull,
    0x938d458b78517f3bull, 0x93a6d95eaf129f88ull, 0x93c071a0eef94bc0ull, 0x93da0e52fcc65b5bull, 0x93f3af759d5cc105ull,
    0x940d550995c19087ull, 0x9426ff0fab1c04b6ull, 0x9440ad88a2b5855dull, 0x945a607541f9ad27ull, 0x947417d64e764f91ull,
    0x948dd3ac8ddb7ed3ull, 0x94a793f8c5fb91d5ull, 0x94c158bbbccb2a1eull, 0x94db21f6386139c4ull, 0x94f4efa8fef70961ull,
    0x950ec1d4d6e83e05ull, 0x9528987a86b2df2cull, 0x9542739ad4f75cb5ull, 0x955c5336887894d5ull, 0x9576374e681bda13ull,
    0x95901fe33ae8f93full, 0x95aa0cf5c80a3f6dull, 0x95c3fe86d6cc7feeull, 0x95ddf4972e9f1a4full, 0x95f7ef2797140053ull,
    0x9611ee38d7dfbbf4ull, 0x962bf1cbb8d9755full, 0x9645f9e101faf8f9ull, 0x966006797b60bd5cull, 0x967a1795ed49e959ull,
    0x96942d3720185a00ull, 0x96ae475ddc50a89full, 0x96c8660aea9a30cbull, 0x96e2893f13bf1665ull, 0x96fcb0fb20ac4ba2ull,
    0x9716dd3fda719714ull, 0x97310e0e0a4199b2ull, 0x974b43667971d4e4ull, 0x97657d49f17ab08eull, 0x977fbbb93bf7811eull,
    0x9799feb522a68d98ull, 0x97b4463e6f6915a7ull, 0x97ce9255ec4357abull, 0x97e8e2fc635c96c9ull, 0x980338329eff2102ull,
    0x981d91f969985541ull, 0x9837f0518db8a96full, 0x9852533bd613b08dull, 0x986cbab90d8020c5ull, 0x988726c9fef7d985ull,
    0x98a1976f7597e995ull, 0x98bc0caa3ca09531ull, 0x98d6867b1f755c24ull, 0x98f104e2e99cffe3ull, 0x990b87e266c189a9ull,
    0x99260f7a62b05097ull, 0x99409baba959ffcfull, 0x995b2c7706d29c96ull, 0x9975c1dd47518c77ull, 0x99905bdf37319b5eull,
    0x99aafa7da2f101c3ull, 0x99c59db957316ac9ull, 0x99e0459320b7fa64ull, 0x99faf20bcc6d5380ull, 0x9a15a324275d9e27ull,
    0x9a3058dcfeb88da9ull, 0x9a4b13371fd166caull, 0x9a65d233581f05e4ull, 0x9a8095d2753be519ull, 0x9a9b5e1544e6227full,
    0x9ab62afc94ff864aull, 0x9ad0fc89338d88fdull, 0x9aebd2bbeeb9599aull, 0x9b06ad9594cfe3d4ull, 0x9b218d16f441d63cull,
    0x9b3c7140dba3a87bull, 0x9b575a1419ada17eull, 0x9b7247917d3bddb2ull, 0x9b8d39b9d54e5538ull, 0x9ba8308df108e21bull,
    0x9bc32c0e9fb34687ull, 0x9bde2c3cb0b93309ull, 0x9bf93118f3aa4cc1ull, 0x9c143aa4383a33a3ull, 0x9c2f48df4e4088b4ull,
    0x9c4a5bcb05b8f443ull, 0x9c6573682ec32c2dull, 0x9c808fb799a2fa19ull, 0x9c9bb0ba16c041bdull, 0x9cb6d67076a7071cull,
    0x9cd200db8a0774caull, 0x9ced2ffc21b5e235ull, 0x9d0863d30eaad9e2ull, 0x9d239c6122031fbaull, 0x9d3ed9a72cffb750ull,
    0x9d5a1ba60105ea29ull, 0x9d75625e6f9f4e03ull, 0x9d90add14a79cb26ull, 0x9dabfdff6367a2a9ull, 0x9dc752e98c5f74c5ull,
    0x9de2ac90977c471full, 0x9dfe0af556fd8b19ull, 0x9e196e189d472420ull, 0x9e34d5fb3ce16e00ull, 0x9e50429e08794336ull,
    0x9e6bb401d2e00343ull, 0x9e872a276f0b98ffull, 0x9ea2a50fb01680f1ull, 0x9ebe24bb693fcfa5ull, 0x9ed9a92b6deb3804ull,
    0x9ef5326091a111adull, 0x9f10c05ba80e5f4full, 0x9f2c531d8504d503ull, 0x9f47eaa6fc7adeacull, 0x9f6386f8e28ba650ull,
    0x9f7f28140b771a79ull, 0x9f9acdf94ba1f493ull, 0x9fb678a97795bf50ull, 0x9fd228256400dd05ull, 0x9feddc6de5b68e13ull,
    0xa0099583d1aef744ull, 0xa0255367fd072836ull, 0xa041161b3d0121bdull, 0xa05cdd9e6703dc4full, 0xa078a9f2509b4e68ull,
    0xa0947b17cf7872f6ull, 0xa0b0510fb9714fc2ull, 0xa0cc2bdae480fbdeull, 0xa0e80b7a26c7a612ull, 0xa103efee568a9b46ull,
    0xa11fd9384a344cf7ull, 0xa13bc758d85457a2ull, 0xa157ba50d79f8939ull, 0xa173b2211eefe793ull, 0xa18faeca8544b6e3ull,
    0xa1abb04de1c28028ull, 0xa1c7b6ac0bb317a8ull, 0xa1e3c1e5da85a361ull, 0xa1ffd1fc25cea188ull, 0xa21be6efc547eefcull,
    0xa23800c190d0cdc4ull, 0xa2541f72606deb8bull, 0xa27043030c496818ull, 0xa28c6b746cb2dbd2ull, 0xa2a898c75a1f5e39ull,
    0xa2c4cafcad298c6aull, 0xa2e102153e918f9eull, 0xa2fd3e11e73d23aeull, 0xa3197ef380379d94ull, 0xa335c4bae2b1f1f0ull,
    0xa3520f68e802bb92ull, 0xa36e5efe69a641f9ull, 0xa38ab37c413e7fe0ull, 0xa3a70ce3489329c7ull, 0xa3c36b345991b47bull,
    0xa3dfce704e4d5ba4ull, 0xa3fc369800ff284cull, 0xa418a3ac4c05f774ull, 0xa43515ae09e6809eull, 0xa4518c9e154b5c5bull,
    0xa46e087d49050ae3ull, 0xa48a894c8009faa0ull, 0xa4a70f0c95768ec4ull, 0xa4c399be648d25deull, 0xa4e02962c8b6206full,
    0xa4fcbdfa9d7fe780ull, 0xa5195786be9ef339ull, 0xa535f60807edd17eull, 0xa552997f556d2c83ull, 0xa56f41ed8343d16eull,
    0xa58bef536dbeb6edull, 0xa5a8a1b1f15103d7ull, 0xa5c55909ea9415cbull, 0xa5e2155c364787cdull, 0xa5fed6a9b15138eaull,
    0xa61b9cf338bd52d8ull, 0xa6386839a9be509bull, 0xa655387de1ad0528ull, 0xa6720dc0be08a20bull, 0xa68ee8031c76be0eull,
    0xa6abc745dac35bdfull, 0xa6c8ab89d6e0f0bdull, 0xa6e594cfeee86b1dull, 0xa70283190119395bull, 0xa71f7665ebd95062ull,
    0xa73c6eb78db5325aull, 0xa7596c0ec55ff55bull, 0xa7766e6c71b34a16ull, 0xa79375d171af828eull, 0xa7b0823ea47b98c2ull,
    0xa7cd93b4e9653569ull, 0xa7eaaa351fe0b69full, 0xa807c5c0278936a1ull, 0xa824e656e020927dull, 0xa8420bfa298f70d1ull,
    0xa85f36aae3e54880ull, 0xa87c6669ef586770ull, 0xa8999b382c45f93full, 0xa8b6d5167b320e08ull, 0xa8d41405bcc7a11bull,
    0xa8f15806d1d89fbdull, 0xa90ea11a9b5defecull, 0xa92bef41fa77771bull, 0xa949427dd06c20f8ull, 0xa9669acefea9e631ull,
    0xa983f83666c5d333ull, 0xa9a15ab4ea7c0ef8ull, 0xa9bec24b6bafe1c7ull, 0xa9dc2efacc6bbc02ull, 0xa9f9a0c3eee13cedull,
    0xaa1717a7b5693979ull, 0xaa3493a70283c30eull, 0xaa5214c2b8d82e5full, 0xaa6f9afbbb351a2full, 0xaa8d2652ec907629ull,
    0xaaaab6c9300789aaull, 0xaac84c5f68defa97ull, 0xaae5e7167a82d430ull, 0xab0386ef48868de0ull, 0xab212beab6a51219ull,
    0xab3ed609a8c0c526ull, 0xab5c854d02e38c03ull, 0xab7a39b5a93ed337ull, 0xab97f344802b95b0ull, 0xabb5b1fa6c2a639aull,
    0xabd375d851e36941ull, 0xabf13edf162675e8ull, 0xac0f0d0f9deb02b0ull, 0xac2ce06ace503970ull, 0xac4ab8f18c9cfb9eull,
    0xac6896a4be3fe929ull, 0xac86798548cf6765ull, 0xaca461941209a7ecull, 0xacc24ed1ffd4af83ull, 0xace0413ff83e5d03ull,
    0xacfe38dee17c7042ull, 0xad1c35afa1ec90fbull, 0xad3a37b3201455b9ull, 0xad583eea42a14ac6ull, 0xad764b55f068f914ull,
    0xad945cf71068ed2full, 0xadb273ce89c6be29ull, 0xadd08fdd43d01491ull, 0xadeeb12425fab15cull, 0xae0cd7a417e474e3ull,
    0xae2b035e015365cdull, 0xae493452ca35b80eull, 0xae676a835aa1d3d5ull, 0xae85a5f09ad65c8eull, 0xaea3e69b733a37d1ull,
    0xaec22c84cc5c9465ull, 0xaee077ad8ef4f136ull, 0xaefec816a3e32456ull, 0xaf1d1dc0f42f61f9ull, 0xaf3b78ad690a4374ull,
    0xaf59d8dcebccce3full, 0xaf783e5065f87af6ull, 0xaf96a908c1373c5dull, 0xafb51906e75b8661ull, 0xafd38e4bc2605522ull,
    0xaff208d83c6933f8ull, 0xb01088ad3fc24479ull, 0xb02f0dcbb6e04583ull, 0xb04d98348c609a49ull, 0xb06c27e8ab09515bull,
    0xb08abce8fdc92bb4ull, 0xb0a957366fb7a3c9ull, 0xb0c7f6d1ec14f496ull, 0xb0e69bbc5e4a20b1ull, 0xb10545f6b1e8f95aull,
    0xb123f581d2ac258full, 0xb142aa5eac77291eull, 0xb161648e2b566bbcull, 0xb18024113b7f401dull, 0xb19ee8e8c94feb08ull,
    0xb1bdb315c14faa74ull, 0xb1dc8299102ebc9full, 0xb1fb5773a2c6672bull, 0xb21a31a66618fe3bull, 0xb23911324751eb91ull,
    0xb257f61833c5b5abull, 0xb276e05918f206e8ull, 0xb295cff5e47db4a3ull, 0xb2b4c4ef8438c65dull, 0xb2d3bf46e61c7cddull,
    0xb2f2befcf84b5954ull, 0xb311c412a9112489ull, 0xb330ce88e6e2f5fbull, 0xb34fde60a05f3b0eull, 0xb36ef39ac44dbe33ull,
    0xb38e0e38419fae17ull, 0xb3ad2e3a076fa4caull, 0xb3cc53a10501aef3ull, 0xb3eb7e6e29c352fbull, 0xb40aaea2654b9840ull,
    0xb429e43ea75b0e47ull, 0xb4491f43dfdbd3edull, 0xb4685fb2fee19e9bull, 0xb487a58cf4a9c180ull, 0xb4a6f0d2b19b34c2ull,
    0xb4c6418526469cbbull, 0xb4e597a54366512eull, 0xb504f333f9de6484ull, 0xb52454323abcab08ull, 0xb543baa0f738c223ull,
    0xb563268120b4179bull, 0xb58297d3a8b9f0d1ull, 0xb5a20e9980ff7205ull, 0xb5c18ad39b63a594ull, 0xb5e10c82e9ef833eull,
    0xb60093a85ed5f76bull, 0xb6202044ec73ea70ull, 0xb63fb259855047d3ull, 0xb65f49e71c1c059aull, 0xb67ee6eea3b22b8full,
    0xb69e89710f17da8dull, 0xb6be316f517c53ccull, 0xb6dddeea5e39002full, 0xb6fd91e328d17791ull, 0xb71d4a5aa4f38816ull,
    0xb73d0851c6773d7full, 0xb75ccbc9815ee876ull, 0xb77c94c2c9d725e8ull, 0xb79c633e9436e656ull, 0xb7bc373dd4ff752eull,
    0xb7dc10c180dc8021ull, 0xb7fbefca8ca41e7cull, 0xb81bd459ed56d882ull, 0xb83bbe70981faec8ull, 0xb85bae0f82542194ull,
    0xb87ba337a1743833ull, 0xb89b9de9eb2a8863ull, 0xb8bb9e27554c3daaull, 0xb8dba3f0d5d920c0ull, 0xb8fbaf4762fb9ee9ull,
    0xb91bc02bf308d161ull, 0xb93bd69f7c8084c1ull, 0xb95bf2a2f60d405full, 0xb97c143756844dbeull, 0xb99c3b5d94e5bff5ull,
    0xb9bc6816a85c7b16ull, 0xb9dc9a63883e3ba1ull, 0xb9fcd2452c0b9deaull, 0xba1d0fbc8b70258full, 0xba3d52ca9e4244e0ull,
    0xba5d9b705c836458ull, 0xba7de9aebe5fea08ull, 0xba9e3d86bc2f4112ull, 0xbabe96f94e73e119ull, 0xbadef6076ddb55b8ull,
    0xbaff5ab2133e45fbull, 0xbb1fc4fa37a07bd9ull, 0xbb4034e0d430ebacull, 0xbb60aa66e249bbacull, 0xbb81258d5b704b6full,
    0xbba1a65539553b63ull, 0xbbc22cbf75d47453ull, 0xbbe2b8cd0af52ee0ull, 0xbc034a7ef2e9fb0cull, 0xbc23e1d62810c7b6ull,
    0xbc447ed3a4f2ea22ull, 0xbc6521786445257dull, 0xbc85c9c560e7b269ull, 0xbca677bb95e6467eull, 0xbcc72b5bfe781bdcull,
    0xbce7e4a795fff8aeull, 0xbd08a39f580c36beull, 0xbd2968444056cafeull, 0xbd4a32974ac54d18ull, 0xbd6b02997368feffull,
    0xbd8bd84bb67ed482ull, 0xbdacb3af106f7adbull, 0xbdcd94c47dcf6049ull, 0xbdee7b8cfb5ebb9full, 0xbe0f6809860993e2ull,
    0xbe305a3b1ae7c7dbull, 0xbe515222b73d15b4ull, 0xbe724fc158792294ull, 0xbe935317fc378237ull, 0xbeb45c27a03fbe90ull,
    0xbed56af142855f66ull, 0xbef67f75e127f1f1ull, 0xbf1799b67a731082ull, 0xbf38b9b40cde6a22ull, 0xbf59df6f970dca35ull,
    0xbf7b0aea17d12021ull, 0xbf9c3c248e2486f8ull, 0xbfbd731ff9304d18ull, 0xbfdeafdd5848fbdfull, 0xbffff25daaef5f4bull,
    0xc0213aa1f0d08db0ull, 0xc04288ab29c5ef5dull, 0xc063dc7a55d54651ull, 0xc08536107530b5e8ull, 0xc0a6956e8836ca8cull,
    0xc0c7fa958f72816bull, 0xc0e965868b9b5028ull, 0xc10ad6427d952c91ull, 0xc12c4cca66709456ull, 0xc14dc91f476a94c3ull,
    0xc16f4b4221ecd277ull, 0xc190d333f78d911full, 0xc1b260f5ca0fbb33ull, 0xc1d3f4889b62e9b4ull, 0xc1f58ded6da36be9ull,
    0xc2172d25431a4f20ull, 0xc238d2311e3d6672ull, 0xc25a7d1201af5281ull, 0xc27c2dc8f03f8940ull, 0xc29de456ecea5db6ull,
    0xc2bfa0bcfad907c8ull, 0xc2e162fc1d61abffull, 0xc3032b1558076350ull, 0xc324f909ae7a42ecull, 0xc346ccda24976407ull,
    0xc368a687be68eba8ull, 0xc38a861380261279ull, 0xc3ac6b7e6e332c95ull, 0xc3ce56c98d21b15dull, 0xc3f047f5e1b04345ull,
    0xc4123f0470cab7b0ull, 0xc4343bf63f8a1ec1ull, 0xc4563ecc5334cb32ull, 0xc4784787b13e5a30ull, 0xc49a56295f47bb30ull,
    0xc4bc6ab2631f37ceull, 0xc4de8523c2c07baaull, 0xc500a57e84549c41ull, 0xc522cbc3ae3220d2ull, 0xc544f7f446dd0a3bull,
    0xc5672a115506daddull, 0xc589621bdf8e9e7dull, 0xc5aba014ed80f22eull, 0xc5cde3fd86180c2eull, 0xc5f02dd6b0bbc3d9ull,
    0xc6127da175019987ull, 0xc634d35edaacbe7eull, 0xc6572f0fe9ae1cd9ull, 0xc67990b5aa245f79ull, 0xc69bf851245bf9eeull,
    0xc6be65e360cf306bull, 0xc6e0d96d68261fb7ull, 0xc70352f04336c51dull, 0xc725d26cfb050663ull, 0xc74857e498c2b9baull,
    0xc76ae35825cfadbbull, 0xc78d74c8abb9b15cull, 0xc7b00c37343c9be8ull, 0xc7d2a9a4c94254fdull, 0xc7f54d1274e2dc84ull,
    0xc817f681416452b2ull, 0xc83aa5f2393b0007ull, 0xc85d5b6667095d4bull, 0xc88016ded5a01b94ull, 0xc8a2d85c8ffe2c45ull,
    0xc8c59fe0a150c915ull, 0xc8e86d6c14f37c14ull, 0xc90b40fff67027b3ull, 0xc92e1a9d517f0ecbull, 0xc950fa453206dcaaull,
    0xc973dff8a41cad1aull, 0xc996cbb8b4041472ull, 0xc9b9bd866e2f27a2ull, 0xc9dcb562df3e8443ull, 0xc9ffb34f140158a9ull,
    0xca22b74c19756bf4ull, 0xca45c15afcc72623ull, 0xca68d17ccb51982dull, 0xca8be7b2929e8414ull, 0xcaaf03fd606664fdull,
    0xcad2265e4290774dull, 0xcaf54ed64732c0c0ull, 0xcb187d667c921885ull, 0xcb3bb20ff1222f62ull, 0xcb5eecd3b38597c8ull,
    0xcb822db2d28dcdffull, 0xcba574ae5d3b4040ull, 0xcbc8c1c762bd56dbull, 0xcbec14fef2727c5cull, 0xcc0f6e561be825b1ull,
    0xcc32cdcdeedada4full, 0xcc5633677b363c5full, 0xcc799f23d11510e5ull, 0xcc9d110400c147eeull, 0xccc089091ab404bcull,
    0xcce407342f95a5f5ull, 0xcd078b86503dcdd1ull, 0xcd2b16008db36a4full, 0xcd4ea6a3f92cbd65ull, 0xcd723d71a40f6535ull,
    0xcd95da6a9ff06444ull, 0xcdb97d8ffe9429b0ull, 0xcddd26e2d1ee9966ull, 0xce00d6642c231462ull, 0xce248c151f8480e3ull,
    0xce4847f6be9552b0ull, 0xce6c0a0a1c07934dull, 0xce8fd2504abcea43ull, 0xceb3a0ca5dc6a55dull, 0xced775796865c0e9ull,
    0xcefb505e7e0af000ull, 0xcf1f317ab256a4c9ull, 0xcf4318cf191918c1ull, 0xcf67065cc65254ffull, 0xcf8afa24ce323a86ull,
    0xcfaef42845188a87ull, 0xcfd2f4683f94eeb5ull, 0xcff6fae5d267018dull, 0xd01b07a2127e56abull, 0xd03f1a9e14fa8316ull,
    0xd06333daef2b2594ull, 0xd0875359b68fef01ull, 0xd0ab791b80d8aa9full, 0xd0cfa52163e54670ull, 0xd0f3d76c75c5db8cull,
    0xd1180ffdccbab67dull, 0xd13c4ed67f345f98ull, 0xd16093f7a3d3a35aull, 0xd184df6251699ac6ull, 0xd1a931179ef7b3c4ull,
    0xd1cd8918a3afb983ull, 0xd1f1e76676f3dcdaull, 0xd2164c023056bcabull, 0xd23ab6ece79b6e4aull, 0xd25f2827b4b585e3ull,
    0xd2839fb3afc91ee1ull, 0xd2a81d91f12ae45aull, 0xd2cca1c391601975ull, 0xd2f12c49a91ea1ddull, 0xd315bd25514d0a2bull,
    0xd33a5457a3029054ull, 0xd35ef1e1b7872c1dull, 0xd38395c4a853978eull, 0xd3a840018f115760ull, 0xd3ccf099859ac379ull,
    0xd3f1a78da5fb0f5eull, 0xd41664df0a6e52aeull, 0xd43b288ecd61919aull, 0xd45ff29e0972c560ull, 0xd484c30dd970e4c9ull,
    0xd4a999df585beca5ull, 0xd4ce7713a164e84cull, 0xd4f35aabcfedfa1full, 0xd51844a8ff8a6409ull, 0xd53d350c4bfe9005ull,
    0xd5622bd6d14018a2ull, 0xd5872909ab75d189ull, 0xd5ac2ca5f6f7d008ull, 0xd5d136acd04f739aull, 0xd5f6471f54376e71ull,
    0xd61b5dfe9f9bce06ull, 0xd6407b4bcf9a03a6ull, 0xd6659f080180ed01ull, 0xd68ac93452d0dcbaull, 0xd6aff9d1e13ba2fdull,
    0xd6d530e1caa49612ull, 0xd6fa6e652d209af2ull, 0xd71fb25d26f62ddcull, 0xd744fccad69d6af4ull, 0xd76a4daf5ac016d6ull,
    0xd78fa50bd239a737ull, 0xd7b502e15c174b7full, 0xd7da67311797f569ull, 0xd7ffd1fc242c61a3ull, 0xd8254343a1772070ull,
    0xd84abb08af4c9e49ull, 0xd870394c6db32c84ull, 0xd895be0ffce309f9ull, 0xd8bb49547d466bacull, 0xd8e0db1b0f798571ull,
    0xd9067364d44a929bull, 0xd92c1232ecb9dea8ull, 0xd951b78679f9cdeaull, 0xd97763609d6ee63eull, 0xd99d15c278afd7b5ull,
    0xd9c2cead2d85854bull, 0xd9e88e21ddeb0d97ull, 0xda0e5421ac0dd383ull, 0xda3420adba4d8704ull, 0xda59f3c72b3c2dccull,
    0xda7fcd6f219e2c0bull, 0xdaa5ada6c06a4d25ull, 0xdacb946f2ac9cc71ull, 0xdaf181c984185df7ull, 0xdb1775b6efe43730ull,
    0xdb3d703891ee17c5ull, 0xdb63714f8e295255ull, 0xdb8978fd08bbd537ull, 0xdbaf874225fe3343ull, 0xdbd59c200a7bac94ull,
    0xdbfbb797daf23755ull, 0xdc21d9aabc52888aull, 0xdc480259d3c01cdeull, 0xdc6e31a64691416cull, 0xdc9467913a4f1c91ull,
    0xdcbaa41bd4b5b6beull, 0xdce0e7473bb40346ull, 0xdd073114956be934ull, 0xdd2d818508324c20ull, 0xdd53d899ba8f1505ull,
    0xdd7a3653d33d3b1aull, 0xdda09ab4792acca9ull, 0xddc705bcd378f7f0ull, 0xdded776e097c13f6ull, 0xde13efc942bba96full,
    0xde3a6ecfa6f27b9aull, 0xde60f4825e0e9123ull, 0xde8780e290313d05ull, 0xdeae13f165af276dull, 0xded4adb0071056a3ull,
    0xdefb4e1f9d1037f1ull, 0xdf21f541509da88bull, 0xdf48a3164adafe78ull, 0xdf6f579fb51e1182ull, 0xdf9612deb8f04420ull,
    0xdfbcd4d4800e8c68ull, 0xdfe39d8234697d00ull, 0xe00a6ce900254e0cull, 0xe031430a0d99e627ull, 0xe0581fe68752e355ull,
    0xe07f037f980fa3feull, 0xe0a5edd66ac34fe0ull, 0xe0ccdeec2a94e111ull, 0xe0f3d6c202df2cf3ull, 0xe11ad5591f30ed37ull,
    0xe141dab2ab4cc8d9ull, 0xe168e6cfd3295d23ull, 0xe18ff9b1c2f146a9ull, 0xe1b71359a7032a53ull, 0xe1de33c8abf1be5full,
    0xe2055afffe83d368ull, 0xe22c8900cbb45d6dull, 0xe253bdcc40b27cddull, 0xe27af9638ae187a0ull, 0xe2a23bc7d7d91225ull,
    0xe2c984fa5564f873ull, 0xe2f0d4fc31856731ull, 0xe3182bce9a6ee4c2ull, 0xe33f8972be8a5a51ull, 0xe366ede9cc751ce6ull,
    0xe38e5934f300f680ull, 0xe3b5cb5561342f2bull, 0xe3dd444c46499618ull, 0xe404c41ad1b08abaull, 0xe42c4ac2330d05e1ull,
    0xe453d8439a37a2daull, 0xe47b6ca0373da88dull, 0xe4a307d93a61129full, 0xe4caa9efd4189a96ull, 0xe4f252e5350fc0faull,
    0xe51a02ba8e26d680ull, 0xe541b9711073052full, 0xe5697709ed3e5987ull, 0xe5913b865607cbb1ull, 0xe5b906e77c8348a8ull,
    0xe5e0d92e9299bb65ull, 0xe608b25cca691616ull, 0xe630927356445b46ull, 0xe658797368b3a716ull, 0xe680675e34743872ull,
    0xe6a85c34ec787a41ull, 0xe6d057f8c3e80ca1ull, 0xe6f85aaaee1fce22ull, 0xe720644c9eb1e4fbull, 0xe74874df0965c84aull,
    0xe7708c6362384954ull, 0xe798aadadd5b9cbeull, 0xe7c0d046af3763d7ull, 0xe7e8fca80c68b5d3ull, 0xe811300029c22912ull,
    0xe8396a503c4bdc68ull, 0xe861ab9979438063ull, 0xe889f3dd161c6093ull, 0xe8b2431c487f6cd8ull, 0xe8da9958464b42aaull,
    0xe902f6924594366cull, 0xe92b5acb7ca45cb8ull, 0xe953c60521fb93b0ull, 0xe97c38406c4f8c56ull, 0xe9a4b17e928bd3daull,
    0xe9cd31c0cbd1dcf4ull, 0xe9f5b9084f79093aull, 0xea1e4756550eb27bull, 0xea46dcac14563418ull, 0xea6f790ac548f464ull,
    0xea981c73a0166dfcull, 0xeac0c6e7dd24392eull, 0xeae97868b50e1557ull, 0xeb1230f760a5f244ull, 0xeb3af09518f3f99bull,
    0xeb63b7431736983full, 0xeb8c850294e287b9ull, 0xebb559d4cba2d79eull, 0xebde35baf558f702ull, 0xec0718b64c1cbddcull,
    0xec3002c80a3c767aull, 0xec58f3f16a3ce6f1ull, 0xec81ec33a6d95a8bull, 0xecaaeb8ffb03ab40ull, 0xecd3f207a1e44b26ull,
    0xecfcff9bd6da4de9ull, 0xed26144dd57b7247ull, 0xed4f301ed9942b84ull, 0xed7853101f27aaeaull, 0xeda17d22e26fe946ull,
    0xedcaae585fddb063ull, 0xedf3e6b1d418a491ull, 0xee1d26307bff4e20ull, 0xee466cd594a722eaull, 0xee6fbaa25b5c8fd5ull,
    0xee990f980da3025bull, 0xeec26bb7e934f213ull, 0xeeebcf032c03ea3dull, 0xef15397b14389349ull, 0xef3eab20e032bc6bull,
    0xef6823f5ce896527ull, 0xef91a3fb1e0ac6e3ull, 0xefbb2b320dbc5e78ull, 0xefe4b99bdcdaf5cbull, 0xf00e4f39cadaad5cull,
    0xf037ec0d176705e5ull, 0xf06190170262e9edull, 0xf08b3b58cbe8b76aull, 0xf0b4edd3b44a4956ull, 0xf0dea788fc110153ull,
    0xf1086879e3fdd149ull, 0xf13230a7ad094509ull, 0xf15c001398638becull, 0xf185d6bee7748280ull, 0xf1afb4aadbdbbc26ull,
    0xf1d999d8b7708cc1ull, 0xf2038649bc42125cull, 0xf22d79ff2c973ed9ull, 0xf25774fa4aeee19cull, 0xf281773c59ffb139ull,
    0xf2ab80c69cb8552aull, 0xf2d5919a563f6f7cull, 0xf2ffa9b8c9f3a685ull, 0xf329c9233b6bae9cull, 0xf353efdaee7653cbull,
    0xf37e1de1271a8390ull, 0xf3a8533729975690ull, 0xf3d28fde3a641a5aull, 0xf3fcd3d79e305b21ull, 0xf4271f2499e3ed7dull,
    0xf45171c6729ef82eull, 0xf47bcbbe6db9fddeull, 0xf4a62d0dd0c5e6e7ull, 0xf4d095b5e18c0b16ull, 0xf4fb05b7e60e3b7bull,
    0xf5257d152486cc2cull, 0xf54ffbcee3689e13ull, 0xf57a81e6695f28bcull, 0xf5a50f5cfd4e8426ull, 0xf5cfa433e6537290ull,
    0xf5fa406c6bc36a4dull, 0xf624e407d52c9f9bull, 0xf64f8f076a560e75ull, 0xf67a416c733f846dull, 0xf6a4fb383821aa85ull,
    0xf6cfbc6c016e0f0bull, 0xf6fa850917cf2f73ull, 0xf7255510c4288238ull, 0xf7502c844f9680beull, 0xf77b0b65036eb12dull,
    0xf7a5f1b4293fb05eull, 0xf7d0df730ad13bb8ull, 0xf7fbd4a2f2243b1eull, 0xf826d1452972cad3ull, 0xf851d55afb304565ull,
    0xf87ce0e5b2094d9bull, 0xf8a7f3e698e3d865ull, 0xf8d30e5efadf36c5ull, 0xf8fe305023541fc8ull, 0xf92959bb5dd4ba74ull,
    0xf9548aa1f62ca7bdull, 0xf97fc30538610c80ull, 0xf9ab02e670b09b77ull, 0xf9d64a46eb939f35ull, 0xfa019927f5bc041full,
    0xfa2cef8adc156270ull, 0xfa584d70ebc5082full, 0xfa83b2db722a033aull, 0xfaaf1fcbbcdd2b40ull, 0xfada944319b12bc9ull,
    0xfb061042d6b28e40ull, 0xfb3193cc4227c3f4ull, 0xfb5d1ee0aa913025ull, 0xfb88b1815ea93210ull, 0xfbb44bafad642efdull,
    0xfbdfed6ce5f09c48ull, 0xfc0b96ba57b7097bull, 0xfc374799525a2a57ull, 0xfc63000b25b6e0efull, 0xfc8ec01121e447bbull,
    0xfcba87ac9733bbaeull, 0xfce656ded630e654ull, 0xfd122da92fa1c7e8ull, 0xfd3e0c0cf486c174ull, 0xfd69f20b761a9eefull,
    0xfd95dfa605d2a15eull, 0xfdc1d4ddf55e88f2ull, 0xfdedd1b496a89f34ull, 0xfe19d62b3bd5c122ull, 0xfe45e2433745695cull,
    0xfe71f5fddb91ba4bull, 0xfe9e115c7b8f884bull, 0xfeca34606a4e63dcull, 0xfef65f0afb18a3caull, 0xff22915d81736f62ull,
    0xff4ecb59511ec8a5ull, 0xff7b0cffbe159675ull, 0xffa756521c8daed1ull, 0xffd3a751c0f7e10bull,
};
// of m in [1 + i/256, 1 + (i+1)/256): the smallest v with v/2^11 (1 + i/256) >= 1,
// and -log2(v/2^11) 2^57
XC_TABLE uint16_t xc_log_inv[256] = {
    2048, 2041, 2033, 2025, 2017, 2009, 2002, 1994, 1986, 1979, 1972, 1964, 1957, 1950, 1942, 1935,
    1928, 1921, 1914, 1907, 1900, 1893, 1886, 1880, 1873, 1866, 1860, 1853, 1847, 1840, 1834, 1827,
    1821, 1815, 1808, 1802, 1796, 1790, 1784, 1778, 1772, 1766, 1760, 1754, 1748, 1742, 1737, 1731,
    1725, 1719, 1714, 1708, 1703, 1697, 1692, 1686, 1681, 1676, 1670, 1665, 1660, 1654, 1649, 1644,
    1639, 1634, 1629, 1624, 1619, 1614, 1609, 1604, 1599, 1594, 1589, 1584, 1580, 1575, 1570, 1566,
    1561, 1556, 1552, 1547, 1543, 1538, 1534, 1529, 1525, 1520, 1516, 1511, 1507, 1503, 1498, 1494,
    1490, 1486, 1482, 1477, 1473, 1469, 1465, 1461, 1457, 1453, 1449, 1445, 1441, 1437, 1433, 1429,
    1425, 1421, 1417, 1414, 1410, 1406, 1402, 1399, 1395, 1391, 1388, 1384, 1380, 1377, 1373, 1369,
    1366, 1362, 1359, 1355, 1352, 1348, 1345, 1341, 1338, 1335, 1331, 1328, 1324, 1321, 1318, 1315,
    1311, 1308, 1305, 1301, 1298, 1295, 1292, 1289, 1286, 1282, 1279, 1276, 1273, 1270, 1267, 1264,
    1261, 1258, 1255, 1252, 1249, 1246, 1243, 1240, 1237, 1234, 1231, 1228, 1225, 1223, 1220, 1217,
    1214, 1211, 1209, 1206, 1203, 1200, 1198, 1195, 1192, 1189, 1187, 1184, 1181, 1179, 1176, 1173,
    1171, 1168, 1166, 1163, 1160, 1158, 1155, 1153, 1150, 1148, 1145, 1143, 1140, 1138, 1135, 1133,
    1130, 1128, 1126, 1123, 1121, 1118, 1116, 1114, 1111, 1109, 1107, 1104, 1102, 1100, 1097, 1095,
    1093, 1090, 1088, 1086, 1084, 1082, 1079, 1077, 1075, 1073, 1070, 1068, 1066, 1064, 1062, 1060,
    1058, 1055, 1053, 1051, 1049, 1047, 1045, 1043, 1041, 1039, 1037, 1035, 1033, 1031, 1029, 1027,
};
XC_TABLE uint64_t xc_log_tab[256] = {
    0x0000000000000000ull, 0x0002876f391a9dc8ull, 0x00056e1588a63197ull, 0x000857a9734f9313ull,
    0x000b4430e855f27aull, 0x000e33b1e91582a0ull, 0x0010c7b844ef1795ull, 0x0013bcdd9b9f00f3ull,
    0x0016b50e297afcceull, 0x001950bcca526da3ull, 0x001beec9151aac2eull, 0x001eef792508b69dull,
    0x002192a5da15c4ecull, 0x0024383deabe0d84ull, 0x0027419ead40d895ull, 0x0029ec74ffe3b484ull,
    0x002c99c4d80ce2adull, 0x002f4992d18c57e6ull, 0x0031fbe3951dd4d4ull, 0x0034b0bbd8996082ull,
    0x003768205f24a728ull, 0x003a2215f965422dull, 0x003cdea185b3eea8ull, 0x003f392bb83a22caull,
    0x0041fa91b28ff78aull, 0x0044be9bd543e257ull, 0x00471f9df778cf6eull, 0x0049e89d59fee11full,
    0x004c4de70b2f8870ull, 0x004f1bed94337943ull, 0x0051858e55ebc0b7ull, 0x005458ae4dbc6d06ull,
    0x0056c6b5f668599bull, 0x005936cb2a70d5a9ull, 0x005c1180c71e7e13ull, 0x005e8614a58d6497ull,
    0x0060fcc133716a9bull, 0x0063758a085012a4ull, 0x0065f072c4f1fb02ull, 0x00686d7f1382d193ull,
    0x006aecb2a7b1d1caull, 0x006d6e113ed2cfbcull, 0x006ff19e9fffd330ull, 0x0072775e9c3b4580ull,
    0x0074ff550e92b572ull, 0x00778985dc42340eull, 0x0079a90fb95cb380ull, 0x007c37606ee803b5ull,
    0x007ec7f6c1d2efdbull, 0x00815ad6bfb3e661ull, 0x008381a9149eb923ull, 0x008618c576ff9e04ull,
    0x0088432546743f30ull, 0x008ade8c15df4bafull, 0x008d0c852eb3a503ull, 0x008fac44b9e43a39ull,
    0x0091dde3262f321bull, 0x0094112ddaf3251full, 0x0096b75a0a91927bull, 0x0098ee5c02d4173aull,
    0x009b271288e64106ull, 0x009dd3cb1fe0fc77ull, 0x00a0104b5f240f66ull, 0x00a24e88af7bec3bull,
    0x00a48e85c70377cfull, 0x00a6d04562324ad2ull, 0x00a913ca43f0a90cull, 0x00ab591735abc725ull,
    0x00ada02f076a607cull, 0x00afe9148fe19e78ull, 0x00b233caac8a52d9ull, 0x00b4805441b686a8ull,
    0x00b6ceb43aa75f41ull, 0x00b91eed89a35b29ull, 0x00bb7103280ce84eull, 0x00bdc4f81679556aull,
    0x00bfa3172c70b441ull, 0x00c1fa72863de1fbull, 0x00c453b5bf2a4e2dull, 0x00c63619aec5cb2eull,
    0x00c892d2eff0efccull, 0x00caf17cda8f8271ull, 0x00ccd83954b63593ull, 0x00cf3a6950f441e0ull,
    0x00d123fba540439aull, 0x00d389bc3d6cbd26ull, 0x00d5762ced6d6df0ull, 0x00d7df88db696424ull,
    0x00d9cee08f2ef08aull, 0x00dc3be2bd8d837full, 0x00de2e2a4492a65dull, 0x00e09eddcfc18b89ull,
    0x00e2941e21dc48d3ull, 0x00e48ab3810b14b4ull, 0x00e700d097aec689ull, 0x00e8fa6bff5fc340ull,
    0x00eaf5626a31ebefull, 0x00ecf1b5b5c12d85ull, 0x00eeef67c386260bull, 0x00f16e7679a82d0bull,
    0x00f36f44b111098eull, 0x00f57177e2a5f156ull, 0x00f7751200c275f9ull, 0x00f97a1501d89ca6ull,
    0x00fb8082e07c57f7ull, 0x00fd885d9b6f2a24ull, 0x00ff91a735abf046ull, 0x01019c61b672d74eull,
    0x0103a88f29557b75ull, 0x0105b6319e4332c1ull, 0x0107c54b2995836cull, 0x0109d5dde41cc6e4ull,
    0x010be7ebeb2cfa18ull, 0x010dfb7760aabbeeull, 0x011010826b187a8full, 0x0111a147ba74653cull,
    0x0113b8f7444275bbull, 0x0115d22c6522ad88ull, 0x0117ece9555fd721ull, 0x011981f9823e8f64ull,
    0x011b9f698381225full, 0x011dbe6788374503ull, 0x011f56ac9ed9a8d2ull, 0x01217868b0c37e7bull,
    0x01239bb9203bcc33ull, 0x012537403a8f2596ull, 0x01275d59f70079abull, 0x0129850e92589b61ull,
    0x012b23e51b39c7b0ull, 0x012d4e6e89164675ull, 0x012eef677ad6fcaeull, 0x01311ccd3590ac3aull,
    0x0132bfee370ee686ull, 0x0134f037d6c5fb24ull, 0x01369586a5706f2full, 0x0138c8bbe0ab6e28ull,
    0x013a703e50fa4df3ull, 0x013c18b41e64d008ull, 0x013e5022fb3a0e98ull, 0x013ffad4e74f1d5eull,
    0x014235429d72a9ddull, 0x0143e236b6a75f73ull, 0x014590247acce3c2ull, 0x01473f0d0d2ec982ull,
    0x01497f209a9b0863ull, 0x014b3056db995a3dull, 0x014ce28bc4549be5ull, 0x014f270b22f5e44eull,
    0x0150db96d04eaa35ull, 0x0152912515c26622ull, 0x015447b7266439aaull, 0x0155ff4e376b8361ull,
    0x0157b7eb8038faf3ull, 0x015a0501e48bd446ull, 0x015bc007cc076f22ull, 0x015d7c18091581e3ull,
    0x015f3933dcb120a2ull, 0x0160f75c8a1b0072ull, 0x0162b69356def7f4ull, 0x016476d98ad99099ull,
    0x01663830703da8d7ull, 0x0167fa99539a2783ull, 0x0169be1583dfc0a4ull, 0x016b82a65266cbe5ull,
    0x016d484d12f52cfaull, 0x016f0f0b1bc44e39ull, 0x0170d6e1c5872d9bull, 0x01729fd26b707c7dull,
    0x017469de6b38d25dull, 0x017635072524f2d2ull, 0x0178014dfc0c271full, 0x0179ceb4555eab8bull,
    0x017b9d3b992c30e3ull, 0x017cd236fba5cc41ull, 0x017ea2a2ed97cce2ull, 0x018074339733a867ull,
    0x018246ea6a6006abull, 0x01841ac8dbc27344ull, 0x0185535771691f09ull, 0x01872925d8cb66acull,
    0x0189001fcdbed999ull, 0x018ad846cf369a41ull, 0x018c13b3791cefffull, 0x018dedd394ee933cull,
    0x018fc924c89ac847ull, 0x0191a5a89dc46b69ull, 0x0192e400f3ff2f96ull, 0x0194c287492c4db0ull,
    0x0196a244683409e2ull, 0x0197e2c542fd71cfull, 0x0199c48be2063c84ull, 0x019ba78d8912825eull,
    0x019cea3e7366be59ull, 0x019ecf50bf43f134ull, 0x01a0136399883a4cull, 0x01a1fa8b145e3adbull,
    0x01a3e2f4ac43f603ull, 0x01a529442d54608full, 0x01a713ca57071aeaull, 0x01a85b83c880d5afull,
    0x01aa482b35ca9cebull, 0x01ab9151be168dd7ull, 0x01ad801f307aa07bull, 0x01aecab6009482abull,
    0x01b0bbae4995d670ull, 0x01b207b89d3bc1ddull, 0x01b3fae09ea5172cull, 0x01b54861bc88149dull,
    0x01b73dbe68b5a1bbull, 0x01b88cb9a2ab5213ull, 0x01b9dc4d0b8ba507ull, 0x01bbd4c8b00b6f25ull,
    0x01bd25daeddc5a84ull, 0x01bf209761c35e3eull, 0x01c0732be1e9feb7ull, 0x01c1c65bdb503ce8ull,
    0x01c3c4488dde1ffaull, 0x01c518ffa9e2cfadull, 0x01c66e54373091e0ull, 0x01c86f7b7ea4a88bull,
    0x01c9c65c26a33233ull, 0x01cb1ddc4196f6d8ull, 0x01cd2248a6c7353bull, 0x01ce7b59ece367cdull,
    0x01cfd50cb182f873ull, 0x01d1dcc8f1282af4ull, 0x01d338120a6dd9d3ull, 0x01d493feb7e8561bull,
    0x01d5f08f93f98892ull, 0x01d74dc539de4f4cull, 0x01d95acc02d690a2ull, 0x01dab9a04e2228eaull,
    0x01dc191b896a324bull, 0x01dd793e53d9200cull, 0x01df8aae0e46f567ull, 0x01e0ec767ccdac60ull,
    0x01e24ee8ae9f0c50ull, 0x01e3b20546f554a1ull, 0x01e515cce9f6a08eull, 0x01e67a403cb6ae6cull,
    0x01e7df5fe538ab35ull, 0x01e9f853f0405beaull, 0x01eb5f254ba8bf06ull, 0x01ecc6a549560785ull,
    0x01ee2ed49397813aull, 0x01ef97b3d5b61552ull, 0x01f10143bbf63308ull, 0x01f26b84f399bd11ull,
    0x01f3d6782ae1fbc3ull, 0x01f5421e11119403ull, 0x01f6ae77566e830dull, 0x01f81b84ac441f24ull,
    0x01f98946c4e51d34ull, 0x01faf7be53ad9b7eull, 0x01fc66ec0d05314eull, 0x01fdd6d0a66103dcull,
};

// (the tables are in device memory where nvcc compiles, so what reads them is
// device code alone there)
#ifdef __CUDACC__
#define XC_TAB(t, i) __ldg(&t[i])
#define XC_TAB_FN __device__ __forceinline__
#else
#define XC_TAB(t, i) t[i]
#define XC_TAB_FN inline
#endif
XC_HD uint64_t xc_mulhi64(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// 2^(k + f / 2^64), |k| <= 1000
XC_TAB_FN double xc_exp2_fixed(int k, uint64_t f) {
  const uint64_t t = XC_TAB(xc_exp2_tab, (uint32_t)(f >> 54));
  const uint64_t Y = xc_mulhi64(f << 10, 0xb17217f7d1cf79abull);   // y 2^74, y = r ln 2 < 2^-10.5
  const uint32_t yh = (uint32_t)(Y >> 32);
  uint32_t p = 0x2aaaaaabu + (xc_mulhi(yh, 0x8888889u) >> 10);       // (1/6 + y/24 + y^2/120) 2^34
  p = 0xaaaaaaabu + (xc_mulhi(yh, p) >> 10);
  const uint64_t y2 = xc_mulhi64(Y, Y);                            // y^2 2^84
  const uint64_t c3 = xc_mulwide((uint32_t)(y2 >> 31), (uint32_t)(xc_mulwide(yh, p) >> 32));   // y^3 (...) 2^97
  const uint64_t E = Y + (y2 >> 11) + (c3 >> 23);                  // (exp(y) - 1) 2^74
  const uint64_t R = t + (xc_mulhi64(t, E) >> 10);
  return xc_from_bits(((uint64_t)(uint32_t)(k + 1022) << 52) + (R >> 11) + ((R >> 10) & 1));
}

XC_TAB_FN double xc_exp(double x) {
  const uint64_t u = xc_bits(x);
  const uint32_t h = (uint32_t)(u >> 32) & 0x7fffffffu;
  if (h < 0x3f100000u) {                                           // |x| < 2^-14: four terms, errors of 2^-75
    const int s = (int)(h >> 20) - 998;                            // Y = |x| 2^77
    const uint64_t m = (u & ((1ull << 52) - 1)) | (1ull << 52);
    const uint64_t Y = s >= 0 ? m << s : (s > -64 ? m >> -s : 0);
    const uint64_t y2 = xc_mulhi64(Y, Y), y3 = xc_mulhi64(y2, Y);  // y^2 2^90, y^3 2^103
    const uint32_t yy = (uint32_t)(y2 >> 32);
    const uint64_t odd = Y + (xc_mulhi64(y3, 0x2aaaaaaaaaaaaaabull) >> 26);
    const uint64_t even = (y2 >> 14) + (xc_mulhi64(xc_mulwide(yy, yy), 0x0aaaaaaaaaaaaaabull) >> 39);
    if ((int64_t)u < 0) {
      const uint64_t E = odd - even;                               // 1 - E 2^-77, half the spacing below 1
      return xc_from_bits(0x3ff0000000000000ull - ((E >> 24) + ((E >> 23) & 1)));
    }
    const uint64_t E = odd + even;
    return xc_from_bits(0x3ff0000000000000ull + (E >> 25) + ((E >> 24) & 1));
  }
  if (h < 0x40862000u) {                                           // |x| < 708
    const uint64_t m = (u << 11) | (1ull << 63);
    const uint64_t H = xc_mulhi64(m, 0xb8aa3b295c17f0bcull), L = m * 0xb8aa3b295c17f0bcull;
    const int s = 1085 - (int)(h >> 20);                           // |x| log2(e) = (H : L) / 2^(s + 64), s >= 53
    int k = s < 64 ? (int)(H >> s) : 0;
    uint64_t f = s < 64 ? (H << (64 - s)) | (L >> s) : (s < 128 ? H >> (s - 64) : 0);
    if ((int64_t)u < 0) {
      k = f == 0 ? -k : -k - 1;
      f = 0 - f;
    }
    return xc_exp2_fixed(k, f);
  }
  return std::exp(x);
}

// log2(x) 2^57 of a normal x in [2^-62, 2^62], to within 2^-56
XC_HD bool xc_log2_ok(double x) { return (uint32_t)(xc_bits(x) >> 52) - 961u <= 123u; }
XC_TAB_FN int64_t xc_log2_fixed(double x) {
  const uint64_t u = xc_bits(x);
  const int k = (int)(u >> 52) - 1023;
  const uint32_t i = (uint32_t)(u >> 44) & 255u;
  const uint64_t R = (((u & ((1ull << 52) - 1)) | (1ull << 52)) * (uint64_t)XC_TAB(xc_log_inv, i) - (1ull << 63)) << 8;
  const uint32_t rh = (uint32_t)(R >> 32);                         // m v = 1 + r, R = r 2^71, r < 2^-7.6
  uint32_t q = 0x55555555u - (xc_mulhi(rh, 0x49249249u) >> 7);     // (1/3 - r/4 + r^2/5 - r^3/6 + r^4/7) 2^33
  q = 0x66666666u - (xc_mulhi(rh, q) >> 7);
  q = 0x80000000u - (xc_mulhi(rh, q) >> 7);
  q = 0xaaaaaaabu - (xc_mulhi(rh, q) >> 7);
  const uint64_t r2 = xc_mulhi64(R, R);                            // r^2 2^78
  const uint64_t c3 = xc_mulwide((uint32_t)(r2 >> 31), (uint32_t)(xc_mulwide(rh, q) >> 31));
  const uint64_t l = R - (r2 >> 8) + (c3 >> 17);                   // log(1 + r) 2^71
  return ((int64_t)k << 57) + (int64_t)XC_TAB(xc_log_tab, i) + (int64_t)(xc_mulhi64(l, 0xb8aa3b295c17f0bcull) >> 13);
}

// 2^(c 2^-58 l 2^-57), l signed: the power of a logarithm above
XC_TAB_FN double xc_exp2_product(uint64_t c, int64_t l) {
  const uint64_t a = l < 0 ? 0 - (uint64_t)l : (uint64_t)l;
  const uint64_t H = xc_mulhi64(a, c), L = a * c;                  // scale 2^115
  int64_t k = (int64_t)(H >> 51);
  uint64_t f = (H << 13) | (L >> 51);
  if (l < 0) {
    k = f == 0 ? -k : -k - 1;
    f = 0 - f;
  }
  if (k < -1000 || k > 1000) return std::exp2((double)k + (double)f * 5.421010862427522e-20);
  return xc_exp2_fixed((int)k, f);
}
