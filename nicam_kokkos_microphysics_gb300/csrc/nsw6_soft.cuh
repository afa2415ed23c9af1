// FP64 quotients, square roots, conversions, exp, log and pow on the integer
// and FP32 pipes.
//
// GB300's FP64 pipe retires one warp instruction per SM every 16 to 19 cycles
// (DFMA 16, DADD 19, a conversion 16, an IEEE division 137, a square root 143,
// measured with 16 warps per SM), its integer and FP32 pipes about two per
// cycle (IMAD, LOP3, SHF 0.5 cycles, IMAD.WIDE 0.7 to 1).  A routine that the
// FP64 pipe needs nine operations for has the time of some 300 integer
// instructions, and these need 40 to 110.  So the step's quotients, roots and
// transcendental functions work on the mantissas as integers here, and the
// FP64 pipe keeps the sums and products.
//
// Quotients and roots are correctly rounded: an approximate quotient (root) to
// well below half a unit, then the exact remainder of the rounded candidate,
// modulo 2^64, decides whether it is the nearest.  exp, log2 and pow work in
// 64-bit fixed point (tables of 2^(j/256) and of log2 of 512 nodes, short
// polynomials), errors below 0.52 units in the last place; a single rounding
// at the end.  Operands and results outside the normal range, infinities and
// NaNs go to the plain FP64 operation (never in a step's ordinary cells; zero
// numerators and radicands, which every absent species gives, are handled
// here).
//
// The larger routines are calls, not inlined: with some forty of them in line
// the FP64 cell kernel had 216 KB of code and waited for instructions 11 of 29
// cycles an instruction; with calls 120 KB, and its time went from 1.03 to
// 0.80 ms (one 16900 x 42 region).
//
// Every routine compiles for the host too, where tests/test_softfp.py compares
// it with the host's IEEE arithmetic and with extended-precision references;
// tests/test_gpu_softfp.py compares the quotients, roots and conversions on the
// device, whose seeds are the special-function unit's.
#pragma once

#include <cmath>
#include <cstdint>

#include "nsw6_fpcmp.cuh"

#ifdef __CUDACC__
#define NSW6_SLOW static __host__ __device__ __noinline__
#define NSW6_CALL static __host__ __device__ __noinline__
#else
#define NSW6_SLOW static inline
#define NSW6_CALL static inline
#endif

namespace nsw6 {

typedef unsigned int u32;
typedef unsigned long long u64;

// ---------------------------------------------------------------- primitives
NSW6_FP_HD u32 soft_umulhi(u32 a, u32 b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (u32)(((u64)a * b) >> 32);
#endif
}
NSW6_FP_HD u32 soft_hi(u64 x) { return (u32)(x >> 32); }
NSW6_FP_HD u64 soft_pair(u32 hi, u32 lo) { return ((u64)hi << 32) | lo; }
// the high word of a 64-bit product, less at most 2 (the low words' product is left out)
NSW6_FP_HD u64 soft_mulhi64(u64 a, u64 b) {
  const u32 ah = soft_hi(a), al = (u32)a, bh = soft_hi(b), bl = (u32)b;
  return (u64)ah * bh + soft_umulhi(ah, bl) + soft_umulhi(al, bh);
}
// bits [s, s + 32) of the word pair hi:lo, s taken modulo 32
NSW6_FP_HD u32 soft_shr(u32 lo, u32 hi, u32 s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_r(lo, hi, s);
#else
  return (u32)(soft_pair(hi, lo) >> (s & 31));
#endif
}
NSW6_FP_HD int soft_clz(u32 x) {
#ifdef __CUDA_ARCH__
  return __clz(x);
#else
  return x ? __builtin_clz(x) : 32;
#endif
}
NSW6_FP_HD float soft_as_float(u32 b) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float f;
  std::memcpy(&f, &b, 4);
  return f;
#endif
}
NSW6_FP_HD u32 soft_float_bits(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  u32 b;
  std::memcpy(&b, &f, 4);
  return b;
#endif
}
// 1 / x and 1 / sqrt(x), the special-function unit's (PTX: rcp.approx.ftz.f32
// within one unit in the last place, rsqrt.approx.ftz.f32 within 2^-22.9
// relative).  The host has them correctly rounded, moved by NSW6_SEED_ULPS
// units (a test sets it) where the device's may be.
#ifndef NSW6_SEED_ULPS
#define NSW6_SEED_ULPS 0
#endif
NSW6_FP_HD float soft_rcp_seed(float x) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return soft_as_float(soft_float_bits(1.0f / x) + (u32)(NSW6_SEED_ULPS));
#endif
}
NSW6_FP_HD float soft_rsqrt_seed(float x) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return soft_as_float(soft_float_bits((float)(1.0 / std::sqrt((double)x))) + (u32)(NSW6_SEED_ULPS));
#endif
}

// An empty call: the block it stands in is branched around, not predicated.
NSW6_SLOW void soft_branch() { asm volatile(""); }

constexpr u64 SOFT_MANT = 0x000FFFFFFFFFFFFFull;
constexpr u64 SOFT_ONE = 0x0010000000000000ull;

// ---------------------------------------------------------------- conversions
NSW6_SLOW float soft_slow_d2f(double x) { return (float)x; }
NSW6_SLOW double soft_slow_f2d(float x) { return (double)x; }

// (float)x, rounded to nearest even
NSW6_FP_HD float soft_d2f(double x) {
  const u64 b = (u64)fp_bits(x);
  const u32 hi = soft_hi(b), lo = (u32)b, ah = hi & 0x7FFFFFFFu;
  // 2^-126 <= |x| < 2^127: drop 29 bits with rounding, exponent bias 1023 -> 127
  if (ah - 0x38100000u < 0x47E00000u - 0x38100000u) {
    const u64 r = soft_pair(ah, lo) + 0x0FFFFFFFull + ((lo >> 29) & 1u);
    return soft_as_float((((u32)(r >> 29)) - 0xC0000000u) | (hi & 0x80000000u));
  }
  if ((ah | lo) == 0u) return soft_as_float(hi);
  return soft_slow_d2f(x);
}
// (double)x
NSW6_FP_HD double soft_f2d(float x) {
  const u32 b = soft_float_bits(x), a = b & 0x7FFFFFFFu;
  if (a - 0x00800000u < 0x7F800000u - 0x00800000u)
    return fp_from_bits((long long)soft_pair(((a >> 3) + 0x38000000u) | (b & 0x80000000u), b << 29));
  if (a == 0u) return fp_from_bits((long long)soft_pair(b, 0u));
  return soft_slow_f2d(x);
}

// ---------------------------------------------------------------- quotients
// The reciprocal of a divisor's mantissa to 32 bits.  m: its 53-bit mantissa;
// r ~ 2^84 / m; e: its exponent field; s: its sign bit (bit 31).
struct SoftDivisor {
  u64 m;
  u32 r;
  int e;   // 0 or 2047: not a normal number
  u32 s;
};

// One Newton step from the special-function unit's reciprocal: with b the top
// 32 bits of m, r0 = 2^32 / b' for a b' 2^-22 above b / 2^31, and
// r = r0 + r0 (1 - b r0) in floor arithmetic is at most 2^63 / b and at least
// that less 3, so r is within 3 of 2^84 / m and below 2^32.  y = 1 / b' has to
// stay below 1, where r0 has its top bit: for b = 2^31 it is 1 - 2^-22, four
// units in the last place below, and the unit is within one.
NSW6_FP_HD SoftDivisor soft_divisor(double b) {
  const u64 bits = (u64)fp_bits(b);
  SoftDivisor d;
  d.m = (bits & SOFT_MANT) | SOFT_ONE;
  d.e = (int)((soft_hi(bits) >> 20) & 0x7FFu);
  d.s = soft_hi(bits) & 0x80000000u;
  const u32 b32 = (u32)(d.m >> 21);                      // [2^31, 2^32)
  const float y = soft_rcp_seed(soft_as_float((b32 >> 8) + 0x3F000002u));   // 1 / (b32 / 2^31 + 2^-22)
  const u32 r0 = (soft_float_bits(fmaxf(y, 0.5f)) << 8) | 0x80000000u;      // y in [0.5, 1)
  const long long err = (long long)(0x8000000000000000ull - (u64)b32 * r0);   // below 2^43 in size
  d.r = r0 + (u32)(int)(((long long)(int)(r0 >> 1) * (long long)(int)(err >> 13)) >> 49);
  return d;
}

NSW6_SLOW double soft_slow_div(double a, double b) { return a / b; }

// The 53-bit mantissa of a / b (both normal), rounded to nearest, as the bits
// of the quotient; *ok: the quotient is a normal number.
NSW6_FP_HD u64 soft_quotient(u64 abits, const SoftDivisor& d, bool& ok) {
  const u32 ahi = soft_hi(abits);
  const int ea = (int)((ahi >> 20) & 0x7FFu);
  u64 ma = (abits & SOFT_MANT) | SOFT_ONE;
  const bool less = ma < d.m;
  if (less) ma <<= 1;                                    // ma / m in [1, 2)
  const u32 q1 = soft_umulhi((u32)(ma >> 22), d.r);      // 2^30 ma / m, to a few units
  const long long r1 = (long long)((ma << 30) - (u64)q1 * d.m);
  // the remainder's quotient, 2^22 r1 / m: r1 / 2^25 fits 32 bits
  const long long q2 = ((long long)(int)(r1 >> 25) * (long long)(int)(d.r >> 1)) >> 36;
  u64 c = ((u64)q1 << 22) + (u64)q2;                     // 2^52 ma / m less between -0.1 and 1.1
  // nearest: c or c + 1 by the remainder 2^52 ma - c m (a quotient is never half way)
  const long long r2 = (long long)((ma << 52) - c * d.m) << 1;
  if (r2 > (long long)d.m) ++c;
  const int e = ea - d.e + 1022 - (less ? 1 : 0);        // exponent field less one (c holds the leading one)
  ok = (u32)(ea - 1) < 2046u && (u32)(d.e - 1) < 2046u && (u32)e < 2045u;
  return c + ((u64)(u32)e << 52) + ((u64)((ahi ^ d.s) & 0x80000000u) << 32);
}

// a / b, correctly rounded
NSW6_CALL double soft_div(double a, SoftDivisor d, double b) {
  const u64 ab = (u64)fp_bits(a);
  bool ok;
  const u64 q = soft_quotient(ab, d, ok);
  if (ok) return fp_from_bits((long long)q);
  if ((ab << 1) == 0ull && (u32)(d.e - 1) < 2046u) return fp_from_bits((long long)(ab ^ ((u64)d.s << 32)));
  return soft_slow_div(a, b);
}
NSW6_CALL double soft_div(double a, double b) { return soft_div(a, soft_divisor(b), b); }
NSW6_CALL double soft_rcp(SoftDivisor d, double b) {
  bool ok;
  const u64 q = soft_quotient(0x3FF0000000000000ull, d, ok);
  return ok ? fp_from_bits((long long)q) : soft_slow_div(1.0, b);
}

// a / b as div_rn's callers form it from a shared reciprocal: a zero over a
// positive b is +0 whatever its sign.
NSW6_SLOW double soft_slow_div_rn(double a, double b) {
  const double rb = 1.0 / b;
  const double q = a * rb;
  return fma(fma(-q, b, a), rb, q);
}
NSW6_CALL double soft_div_rn(double a, SoftDivisor d, double b) {
  const u64 ab = (u64)fp_bits(a);
  // first, as whole warps divide the zeros of a species they do not hold
  if ((ab << 1) == 0ull && d.s == 0u && (u32)(d.e - 1) < 2046u) return 0.0;
  bool ok;
  const u64 q = soft_quotient(ab, d, ok);
  return ok ? fp_from_bits((long long)q) : soft_slow_div_rn(a, b);
}

// ---------------------------------------------------------------- square root
NSW6_SLOW double soft_slow_sqrt(double x) { return std::sqrt(x); }

// sqrt(x), correctly rounded: s = sqrt(M) of the mantissa scaled to
// M in [2^62, 2^64), to the nearest 32-bit number by one Newton step from the
// special-function unit's reciprocal root, c = 2^21 sqrt(M) from the remainder
// M - s^2, then the exact remainder of the candidate c.
NSW6_CALL double soft_sqrt(double x) {
  const u64 b = (u64)fp_bits(x);
  const u32 hi = soft_hi(b);
  if (hi - 0x00100000u >= 0x7FE00000u) {   // not positive and normal
    if ((b << 1) == 0ull) return x;
    return soft_slow_sqrt(x);
  }
  const int e = (int)(hi >> 20) - 1023;
  const u64 M = ((b & SOFT_MANT) | SOFT_ONE) << (10 + (e & 1));   // f 2^62, f in [1, 2) (e even) or [2, 4)
  const u32 mh = soft_hi(M);                             // f 2^30
  const u32 odd = mh >> 31;                              // f >= 2: its float has the higher exponent
  const float f = soft_as_float(odd ? (((mh >> 8) & 0x007FFFFFu) | 0x40000000u)
                                    : (((mh >> 7) & 0x007FFFFFu) | 0x3F800000u));
  // 2^31 / sqrt(f), below 2^31 (the unit may give more than 1 for f = 1)
  const int y = (int)(fminf(soft_rsqrt_seed(f), 1.0f) * 2147483520.0f);
  const u64 p = (u64)mh * (u32)y;                        // 2^61 sqrt(f)
  u32 s = (p >> 62) ? 0xFFFFFFFFu : (u32)(p >> 30);      // 2^31 sqrt(f) to 2^11
  long long r = (long long)(M - (u64)s * s);             // below 2^44 in size
  // r / (2 s) = r y / 2^63, to the nearest
  s += (u32)(int)(((long long)(int)(r >> 14) * (long long)y + (1ll << 48)) >> 49);
  s = s < 0x80000000u ? 0xFFFFFFFFu : s;                 // 2^32 wrapped around
  r = (long long)(M - (u64)s * s);                       // below 2^34 in size
  // c = 2^21 s + 2^21 r / (2 s), to the nearest; within 1.2 of the root
  u64 c = ((u64)s << 21) + (u64)(((long long)(int)(r >> 6) * (long long)y + (1ll << 35)) >> 36);
  // nearest: M 2^42 against (c +- 1/2)^2
  const long long t = (long long)((M << 42) - c * c);
  if (t > (long long)c) {
    ++c;
  } else if (t <= -(long long)c) {
    --c;
  }
  return fp_from_bits((long long)(c + ((u64)(u32)((e >> 1) + 1022) << 52)));
}

// ---------------------------------------------------------------- exp, log, pow
// Tables: t[256]: 2^(j/256) in units of 2^-63; lt[512]: -log2(n_j) in units of
// 2^-64; ic[512]: n_j 2^15, n_j the least multiple of 2^-15 with m n_j >= 1
// for every m in [1 + j/512, 1 + (j+1)/512).
constexpr int SOFT_EXP_N = 256, SOFT_LOG_N = 512;
struct SoftTables {
  const u64* t;
  const u64* lt;
  const unsigned short* ic;
};

// 2^(k + f / 2^64), rounded to nearest (k + f / 2^64 in the normal range's
// exponents).  The table's entry at the top 8 bits of f, r the rest (r < 2^-8):
// 2^r - 1 = r (c1 + r (c2 + r (c3 + r (c4 + r c5)))) with the Taylor
// coefficients ln2^n / n! (the next term is below 2^-60).  r has 56 bits, the
// terms from c3 on are below 2^-24 of the result and take 32-bit products.
NSW6_FP_HD double soft_exp2(int k, u64 f, const u64* T) {
  const u64 t = T[f >> 56];
  const u64 R = f << 8;                                  // r 2^72
  const u32 r = soft_hi(R);                              // r 2^40
  const u32 s4 = 660952799u + (soft_umulhi(r, 91627513u) >> 8);           // 2^36 (c4 + r c5)
  const u32 s3 = 3814213304u + (soft_umulhi(r, s4) >> 8);                 // 2^36 (c3 + ...)
  const u64 s2 = 0x3D7F7BFF058B1D50ull + (((u64)r * s3) >> 12);           // 2^64 (c2 + ...)
  const u64 s1 = 0xB17217F7D1CF79ABull + (soft_mulhi64(R, s2) >> 8);      // 2^64 (c1 + ...)
  const u64 M = t + (soft_mulhi64(t, soft_mulhi64(R, s1)) >> 8);          // 2^63 2^(f / 2^64)
  // (M + 0x400 would run over for M next to 2^64)
  return fp_from_bits((long long)((M >> 11) + ((u32)(M >> 10) & 1u) + ((u64)(u32)(k + 1022) << 52)));
}

// Words 1 to 3 of p >> s (p the 128-bit number w3:w2:w1:w0, 32 <= s <= 127):
// the 64-bit fraction and, as the result, what stands above it.
NSW6_FP_HD u32 soft_shift_fixed(u32 w1, u32 w2, u32 w3, int s, u64& f) {
  const int ws = s >> 5;
  const u32 a0 = ws == 1 ? w1 : ws == 2 ? w2 : w3;
  const u32 a1 = ws == 1 ? w2 : ws == 2 ? w3 : 0u;
  const u32 a2 = ws == 1 ? w3 : 0u;
  f = soft_pair(soft_shr(a1, a2, (u32)s), soft_shr(a0, a1, (u32)s));
  return a2 >> (s & 31);
}

NSW6_SLOW double soft_slow_exp(double x) { return std::exp(x); }

// exp(x) = 2^(x log2 e) for |x| < 708, the product with 96 bits of log2 e.
NSW6_CALL double soft_exp(double x, SoftTables T) {
  const u64 b = (u64)fp_bits(x);
  const u32 ah = soft_hi(b) & 0x7FFFFFFFu;
  if (ah >= 0x40862000u) return soft_slow_exp(x);        // 708, infinities, NaN
  // |x| = m 2^(e - 63), m in [2^63, 2^64); words 1 .. 3 of m (log2 e 2^63)
  const int e = (int)(ah >> 20) - 1023;
  const u64 m = ((b & SOFT_MANT) | SOFT_ONE) << 11;
  const u32 mh = soft_hi(m), ml = (u32)m;
  const u64 A = (u64)mh * 0x5C17F0BBu + soft_umulhi(ml, 0x5C17F0BBu);
  const u64 B = (u64)ml * 0xB8AA3B29u + soft_umulhi(mh, 0xBE87FED0u);
  const u64 C = (u64)(u32)A + (u32)B;
  const u64 top = (u64)mh * 0xB8AA3B29u + soft_hi(A) + soft_hi(B) + soft_hi(C);
  // |x| log2 e = product 2^(e - 126); fraction in units of 2^-64.  A zero or subnormal x
  // has its bits shifted out.
  const int s = 62 - e > 127 ? 127 : 62 - e;             // 53 at least
  u64 f;
  int k = (int)soft_shift_fixed((u32)C, (u32)top, soft_hi(top), s, f);
  if (b >> 63) {
    f = 0ull - f;
    k = -k - (f != 0ull ? 1 : 0);
  }
  return soft_exp2(k, f, T.t);
}

// log2 of a positive normal x as I + F / 2^64 (F to a few units): the exponent,
// the table's log2 of the node and log2(1 + r), r = m n_j - 1 < 2^-8.8, by
// r (C1 - r (C2 - r (C3 - ... r C6))), C_n = 1 / (n ln2) (the next term is
// below 2^-64).
NSW6_FP_HD int soft_log2(u64 b, const SoftTables& T, u64& F) {
  const u64 m = (b & SOFT_MANT) | SOFT_ONE;
  const u32 j = (u32)(b >> 43) & (SOFT_LOG_N - 1);
  const u64 R = (m * T.ic[j]) << 5;                      // r 2^72: m n_j 2^67 less 2^67, which is 0 modulo 2^64
  const u32 r = soft_hi(R);                              // r 2^40
  const u32 g5 = 0x93BB6287u - (soft_umulhi(r, 0x7B1C2770u) >> 8);        // 2^33 (C5 - r C6)
  const u32 g4 = 0xB8AA3B29u - (soft_umulhi(r, g5) >> 8);                 // 2^33 (C4 - ...)
  const u64 g3 = 0x7B1C2770E80FF5D2ull - (((u64)r * g4) >> 9);            // 2^64 (C3 - ...)
  const u64 g2 = 0xB8AA3B295C17F0BBull - (soft_mulhi64(R, g3) >> 8);      // 2^64 (C2 - ...)
  const u64 g1 = 0xB8AA3B295C17F0BBull - (soft_mulhi64(R, g2) >> 9);      // 2^63 (C1 - ...)
  F = T.lt[j] + (soft_mulhi64(R, g1) >> 7);
  return (int)(b >> 52) - 1023;
}

NSW6_SLOW double soft_slow_log(double x) { return std::log(x); }

// log(x) for x positive and normal, away from 1 (|x - 1| >= 2^-7: the
// logarithm's error is one of 2^-62 absolute): log2(x) ln2, normalised.
NSW6_CALL double soft_log(u64 b, SoftTables T) {
  u64 f;
  const int I = soft_log2(b, T, f);
  u32 i = (u32)I;
  if (I < 0) {
    f = 0ull - f;
    i = (u32)(-I) - (f != 0ull ? 1u : 0u);
  }
  // the leading 64 bits, of which the first weighs 2^(31 - z)
  u32 w2 = i, w1 = soft_hi(f), w0 = (u32)f;
  int z = 0;
  if (w2 == 0u) { w2 = w1; w1 = w0; w0 = 0u; z = 32; }
  const u32 l = (u32)soft_clz(w2);                       // below 32: |log2 x| > 2^-7
  z += (int)l;
  const u64 m = soft_pair(soft_shr(w1, w2, 32u - l), soft_shr(w0, w1, 32u - l));
  const u64 mm = l ? m : soft_pair(w2, w1);              // (a shift by 32 is one by 0)
  u64 p = soft_mulhi64(mm, 0xB17217F7D1CF79ABull);
  if (!(p >> 63)) { p <<= 1; ++z; }
  // (p + 0x400 would run over for p next to 2^64, a logarithm just below a
  // power of two; rounded so, the carry goes into the exponent)
  return fp_from_bits((long long)(((p >> 11) + ((u32)(p >> 10) & 1u) + ((u64)(u32)(31 - z + 1022) << 52)) |
                                  ((u64)((u32)I & 0x80000000u) << 32)));
}

NSW6_SLOW double soft_slow_pow(double x, double y) { return std::pow(x, y); }

// x^y = 2^(y log2 x) for x positive and normal, 2^-33 <= |y| < 2^7 and
// |y log2 x| < 1021: the product to 2^-60 absolute.
NSW6_CALL double soft_pow(double x, double y, SoftTables T) {
  const u64 xb = (u64)fp_bits(x), yb = (u64)fp_bits(y);
  const u32 xh = soft_hi(xb), yh = soft_hi(yb) & 0x7FFFFFFFu;
  if (xh - 0x00100000u >= 0x7FE00000u || yh - 0x3DE00000u >= 0x40600000u - 0x3DE00000u) return soft_slow_pow(x, y);
  u64 F;
  const int I = soft_log2(xb, T, F);
  const u64 Y = ((yb & SOFT_MANT) | SOFT_ONE) << 11;     // |y| = Y 2^(ey - 63)
  const int ey = (int)(yh >> 20) - 1023;
  // (I 2^64 + F) Y / 2^64 = w2:w1:w0, a signed 96-bit number
  const u64 V = soft_mulhi64(F, Y);
  const u64 lo = (u64)(u32)I * (u32)Y + V;               // carries out of 64 bits: see c
  const u32 c = lo < V ? 1u : 0u;
  const u64 hi = (u64)(u32)I * soft_hi(Y) + soft_hi(lo) + ((u64)c << 32) - (I < 0 ? Y : 0ull);
  // times 2^(ey + 1) (y log2 x in units of 2^-64), negated for y < 0
  u32 w0 = (u32)lo, w1 = (u32)hi, w2 = soft_hi(hi);
  if (yb >> 63) {
    const u64 n = 0ull - soft_pair(w1, w0);
    w2 = ~w2 + (n == 0ull ? 1u : 0u);
    w1 = soft_hi(n);
    w0 = (u32)n;
  }
  const int s = ey + 1;                                  // -32 .. 7
  u64 f;
  int k;
  if (s >= 0) {
    if (s != 0) {
      // what the shift moves out of the top word must be sign bits: checked with k's range below
      const u32 t = 32u - (u32)s;
      const int top = (int)w2 >> (31 - s);
      if (top != 0 && top != -1) return soft_slow_pow(x, y);
      w2 = soft_shr(w1, w2, t);
      w1 = soft_shr(w0, w1, t);
      w0 = w0 << s;
    }
  } else if (s > -32) {
    w0 = soft_shr(w0, w1, (u32)-s);
    w1 = soft_shr(w1, w2, (u32)-s);
    w2 = (u32)((int)w2 >> -s);
  } else {
    w0 = w1;
    w1 = w2;
    w2 = (u32)((int)w2 >> 31);
  }
  f = soft_pair(w1, w0);
  k = (int)w2;
  if ((u32)(k + 1021) >= 2042u) return soft_slow_pow(x, y);
  return soft_exp2(k, f, T.t);
}

}  // namespace nsw6
