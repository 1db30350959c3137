// Exactly rounded FP64 results built with integer arithmetic (the FP64 pipe of
// this GPU retires ~2 operations per clock per SM; integer multiplies and
// shifts run far wider).  Host and device share these definitions, so the
// CPU tests check the very code the kernels run against IEEE arithmetic.
#pragma once

#include <stdint.h>
#include <string.h>

#include <cmath>

#if defined(__CUDACC__)
#define A4G_HD __host__ __device__ __forceinline__
#else
#define A4G_HD inline
#endif

namespace a4g {

A4G_HD int clz64(unsigned long long x) {
#if defined(__CUDA_ARCH__)
  return __clzll((long long)x);
#else
  return x ? __builtin_clzll(x) : 64;
#endif
}
A4G_HD unsigned long long bits_of(double x) {
#if defined(__CUDA_ARCH__)
  return (unsigned long long)__double_as_longlong(x);
#else
  unsigned long long u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
A4G_HD double double_of(unsigned long long u) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)u);
#else
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}
// The double nearest (ties to even) to u * 2^e2 with sign `neg`, u an
// unsigned 64-bit magnitude, rounded once: to 53 bits in the normal range, to
// a multiple of 2^-1074 below it (subnormal results and zero), to infinity
// beyond the largest double.
A4G_HD double u64_scaled_to_double(unsigned long long u, bool neg, int e2) {
  if (u == 0) return 0.0;
  const unsigned long long sbit = neg ? (1ull << 63) : 0ull;
  const int nbits = 64 - clz64(u);
  if (e2 + nbits - 1 < -1022) {  // below 2^-1022: the unit is 2^-1074
    const int sh = -1074 - e2;    // bits of u below the unit
    unsigned long long q;
    if (sh <= 0) {
      q = u << (-sh);  // exact: a multiple of the unit below 2^-1022
    } else if (sh > 64) {
      q = 0;  // below half a unit
    } else {
      q = sh == 64 ? 0ull : u >> sh;
      const unsigned long long rem = sh == 64 ? u : u & ((1ull << sh) - 1), half = 1ull << (sh - 1);
      if (rem > half || (rem == half && (q & 1ull))) ++q;
    }
    return double_of(sbit | q);  // q = 2^52 (rounded up to the least normal) has the right bits too
  }
  unsigned long long mant;
  int e = e2;
  if (nbits <= 53) {
    mant = u << (53 - nbits);
    e -= 53 - nbits;
  } else {
    const int sh = nbits - 53;
    mant = u >> sh;
    const unsigned long long rem = u & ((1ull << sh) - 1), half = 1ull << (sh - 1);
    if (rem > half || (rem == half && (mant & 1ull))) ++mant;
    e += sh;
    if (mant == (1ull << 53)) mant >>= 1, ++e;
  }
  const int field = e + 52 + 1023;  // value = mant * 2^e, mant in [2^52, 2^53)
  if (field > 2046) return double_of(sbit | 0x7FF0000000000000ull);
  return double_of(sbit | ((unsigned long long)field << 52) | (mant & ((1ull << 52) - 1)));
}

// (neg ? -1 : 1) * v * 2^e2 rounded once to the nearest double (ties to
// even), v a signed 64-bit integer: normalise, keep 53 bits, round on the 11
// below, and build the bits by one addition (a mantissa that rounds up to
// 2^53 carries into the exponent field).  Branch-free for results in the
// normal range; the rest takes u64_scaled_to_double.  Same bits as negating
// the result of u64_scaled_to_double (a zero keeps the sign the negation
// gives it).
A4G_HD double i64_scaled_to_double(long long v, int e2, bool neg) {
#if defined(__CUDA_ARCH__)
  // On the GPU the integer-to-FP64 conversion rounds v once to 53 bits (to
  // nearest, ties to even), and the scaling by 2^e2 is an exact addition to
  // the exponent field while the result stays normal: the same bits as the
  // integer construction below, in three instructions.
  if (v != 0) {
    const unsigned long long b = bits_of(__ll2double_rn(v));
    const int field = int((b >> 52) & 0x7FF) + e2;
    if (field >= 1 && field <= 2046)
      return double_of((b + ((unsigned long long)(long long)e2 << 52)) ^ (neg ? (1ull << 63) : 0ull));
  }
#endif
  const unsigned long long sign = (v < 0) != neg ? (1ull << 63) : 0ull;
  const unsigned long long u = v < 0 ? (unsigned long long)(-v) : (unsigned long long)v;
  const int n = clz64(u | 1ull);  // u = 0 is mapped to a signed zero at the end
  const unsigned long long norm = u << n;  // leading one at bit 63
  unsigned long long mant = norm >> 11;    // 53 bits, leading one at bit 52
  const unsigned long long rem = norm & 0x7FFull;
  mant += (rem > 0x400ull || (rem == 0x400ull && (mant & 1ull))) ? 1ull : 0ull;
  const int field = e2 + 63 - n + 1023;  // biased exponent of the leading one
  if (u != 0 && (field < 1 || field > 2045)) return u64_scaled_to_double(u, sign != 0, e2);
  const unsigned long long bits =
      u ? sign | ((((unsigned long long)(field - 1)) << 52) + mant) : (neg ? (1ull << 63) : 0ull);
  return double_of(bits);
}

#if defined(__CUDACC__)
// v * 2^e2 rounded once, branch-free: valid (the return value) for v != 0 and
// a normal result; the same bits as i64_scaled_to_double there.
__device__ __forceinline__ bool i64_scaled_normal(long long v, int e2, double* x) {
  const unsigned long long b = bits_of(__ll2double_rn(v));
  const int field = int((b >> 52) & 0x7FF) + e2;
  *x = double_of(b + ((unsigned long long)(long long)e2 << 52));
  return v != 0 && uint32_t(field - 1) < 2046u;
}
#endif

// The same for a two's-complement 128-bit integer N.
A4G_HD double i128_scaled_to_double(__int128 N, int e2) {
  const bool neg = N < 0;
  const unsigned __int128 u = neg ? (unsigned __int128)(-N) : (unsigned __int128)N;
  const unsigned long long hi = (unsigned long long)(u >> 64);
  if (hi == 0) return u64_scaled_to_double((unsigned long long)u, neg, e2);
  // keep the top 63 bits and fold the rest into a sticky bit below them (the
  // rounding position lies above it, so the rounding is exact)
  const int sh = 65 - clz64(hi);  // u >> sh has 63 bits
  const unsigned long long top = (unsigned long long)(u >> sh);
  const bool sticky = (u & ((((unsigned __int128)1) << sh) - 1)) != 0;
  return u64_scaled_to_double((top << 1) | (sticky ? 1ull : 0ull), neg, e2 + sh - 1);
}

A4G_HD uint32_t mulhi32(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __umulhi(a, b);
#else
  return uint32_t(((unsigned long long)a * b) >> 32);
#endif
}
A4G_HD float float_of(uint32_t u) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(u);
#else
  float x;
  memcpy(&x, &u, 4);
  return x;
#endif
}
A4G_HD uint32_t bits_of(float x) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(x);
#else
  uint32_t u;
  memcpy(&u, &x, 4);
  return u;
#endif
}
// 1/x, 1 < x < 2, to within one unit in the last place (the GPU's approximate
// reciprocal; on the host the nearest float, or A4G_RCP_ULP units off it, so
// that a test can show that the division needs no more than this)
A4G_HD float rcp_approx(float x) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
#ifndef A4G_RCP_ULP
#define A4G_RCP_ULP 0
#endif
  return float_of(bits_of(1.0f / x) + uint32_t(A4G_RCP_ULP));
#endif
}

// a / b rounded to the nearest double (ties to even; a quotient of two
// doubles is never exactly halfway) where a, b and the quotient are normal
// numbers; the return value says whether it is valid.  Branch-free, so that a
// kernel can run several divisions interleaved (the FP64 pipe of this GPU
// takes 5 clocks per division and SM).
//
// With significands ma, mb in [2^52, 2^53) and A = ma or 2 ma (doubled when ma
// < mb, so that v = A 2^52 / mb lies in [2^52, 2^53)), the result's
// significand is RN(v).  Two quotient digits are estimated through a 31-bit
// reciprocal and the exact remainder decides the rounding (Knuth, TAOCP vol.
// 2, 4.3.1: a digit's estimate, then continue from the remainder):
//  1. R ~ R* = 2^83 / mb, 2^30 < R* <= 2^31: the FP32 reciprocal of f = mb's
//     top 24 bits with the last two set (f in (1 + 2^-22, 2), so 1/f + 1 lies
//     below 2 and its fraction field is 2^23 / f; relative error below
//     2^-20.6), then one Newton-Raphson step R + R (1 - R / R*) in 32-bit
//     integers on mb's top 32 bits: with t = floor(m32 R / 2^32) and
//     e = 2^30 - 2 - t, |e| <= 640, R += ((R >> 10) e) >> 20 lands in
//     (R* - 5.1, R* - 0.9).
//  2. q1 = floor((A >> 22) R / 2^32) lies in (A 2^29 / mb - 6.6, A 2^29 / mb],
//     so s1 = A 2^29 - q1 mb (exact in wrapping 64-bit arithmetic) in
//     [0, 6.6 mb), below 2^56.
//  3. h = floor((s1 >> 24) R / 2^32) lies in (16 w - 5.7, 16 w] with
//     w = s1 2^23 / mb = v - q1 2^23; m0 = q1 2^23 + ((h + 10) >> 4) is within
//     0.67 of v.
//  4. r = A 2^52 - m0 mb, |r| < 0.67 mb, exact in wrapping 64-bit arithmetic:
//     RN(v) = m0 + 1 where 2 r > mb, m0 - 1 where 2 r < -mb, else m0.
A4G_HD bool div_rn_int(double a, double b, double* q) {
  const unsigned long long ua = bits_of(a), ub = bits_of(b);
  const uint32_t ah = uint32_t(ua >> 32), bh = uint32_t(ub >> 32);
  const unsigned long long mb = (ub & ((1ull << 52) - 1)) | (1ull << 52);
  unsigned long long A = (ua & ((1ull << 52) - 1)) | (1ull << 52);
  const int adj = A < mb ? 1 : 0;
  A += adj ? A : 0ull;  // [mb, 2 mb)
  const float f = float_of(0x3F800000u | (uint32_t(mb >> 29) & 0x7FFFFFu) | 3u);
  uint32_t R = (bits_of(rcp_approx(f) + 1.0f) & 0x7FFFFFu) << 8;
  const int e = int((1u << 30) - 2u - mulhi32(uint32_t(mb >> 21), R));
  R += uint32_t((int(R >> 10) * e) >> 20);
  const uint32_t q1 = mulhi32(uint32_t(A >> 22), R);
  const unsigned long long s1 = (A << 29) - (unsigned long long)q1 * mb;
  const uint32_t h = mulhi32(uint32_t(s1 >> 24), R);
  const unsigned long long m0 = (unsigned long long)q1 * (1u << 23) + ((h + 10u) >> 4);
  const long long r2 = (long long)(((A << 52) - m0 * mb) << 1);
  const uint32_t up = uint32_t((unsigned long long)((long long)mb - r2) >> 63);
  const uint32_t down = uint32_t((unsigned long long)((long long)mb + r2) >> 63);
  // the exponents and the sign in the high word: field = ea - eb + 1023 - adj,
  // one less because the significand's leading bit adds one
  const int ea = int((ah >> 20) & 0x7FFu), eb = int((bh >> 20) & 0x7FFu);
  const int field = ea - eb + 1023 - adj;
  const uint32_t high = (uint32_t(field - 1) << 20) + ((ah ^ bh) & 0x80000000u);
  const unsigned long long bits = m0 + (((unsigned long long)high << 32) + up - down);
  *q = double_of(bits);
  return uint32_t(ea - 1) < 2046u && uint32_t(eb - 1) < 2046u && uint32_t(field - 1) < 2045u;
}

// a / b rounded to the nearest double: div_rn_int where it applies, the FP64
// divide otherwise (zero, subnormal or non-finite operands or results).
A4G_HD double div_rn_slow(double a, double b) {
#if defined(__CUDA_ARCH__)
  return __ddiv_rn(a, b);
#else
  return a / b;
#endif
}
A4G_HD double div_rn(double a, double b) {
  double q;
  return div_rn_int(a, b, &q) ? q : div_rn_slow(a, b);
}

// N quotients a[i] / b[i], their steps interleaved; the rare operands that
// div_rn_int does not take go through the FP64 divide afterwards.
template <int N>
A4G_HD void div_rn_n(const double (&a)[N], const double (&b)[N], double (&q)[N]) {
  bool ok[N], all = true;
#pragma unroll
  for (int i = 0; i < N; ++i) ok[i] = div_rn_int(a[i], b[i], &q[i]), all = all && ok[i];
  if (all) return;
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (!ok[i]) q[i] = div_rn_slow(a[i], b[i]);
}

// x != 0 without the FP64 pipe
A4G_HD bool nonzero(double x) { return (bits_of(x) << 1) != 0ull; }

}  // namespace a4g
