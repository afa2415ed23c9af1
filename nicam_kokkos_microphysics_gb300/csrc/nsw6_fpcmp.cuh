// IEEE-754 double comparisons evaluated on the integer pipe.
//
// On GB300 an FP64 compare issues to the FP64 pipe, which completes about two
// operations per SM per cycle, while the integer pipe completes 64; the NSW6
// kernels are FP64-pipe bound, so their comparisons (min / max, thresholds,
// range checks) are computed from the bit patterns instead.  Each function
// returns exactly what the IEEE comparison returns for every pair of doubles:
// false when either operand is NaN, -0 equal to +0.
//
// For a non-NaN x with bits b (as a signed 64-bit integer), the key
// b ^ ((b >> 63) & 0x7FF...F) orders the doubles like the reals, except that
// -0 (key -1) sorts below +0 (key 0); the zero pair is tested separately.
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define NSW6_FP_HD __host__ __device__ __forceinline__
#else
#define NSW6_FP_HD inline
#endif

namespace nsw6 {

constexpr long long FP_ABS = 0x7FFFFFFFFFFFFFFFll;   // all but the sign
constexpr long long FP_INF = 0x7FF0000000000000ll;   // +inf; larger magnitudes are NaN

NSW6_FP_HD long long fp_bits(double x) {
#ifdef __CUDA_ARCH__
  return __double_as_longlong(x);
#else
  long long b;
  std::memcpy(&b, &x, sizeof b);
  return b;
#endif
}

// The two words of a double, and the double of two words.  Where one word
// decides, or each by itself, the forms below go by words: of the same test on
// the 64-bit pattern the compiler makes an FP64 instruction, 16 to 19 cycles of
// an SM's FP64 pipe (see each).
NSW6_FP_HD unsigned fp_hi(double x) {
#ifdef __CUDA_ARCH__
  return (unsigned)__double2hiint(x);
#else
  return (unsigned)((unsigned long long)fp_bits(x) >> 32);
#endif
}
NSW6_FP_HD unsigned fp_lo(double x) {
#ifdef __CUDA_ARCH__
  return (unsigned)__double2loint(x);
#else
  return (unsigned)fp_bits(x);
#endif
}
NSW6_FP_HD double fp_of_words(unsigned hi, unsigned lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)hi, (int)lo);
#else
  const unsigned long long b = ((unsigned long long)hi << 32) | lo;
  double x;
  std::memcpy(&x, &b, sizeof x);
  return x;
#endif
}

NSW6_FP_HD long long fp_key(long long b) { return b ^ ((b >> 63) & FP_ABS); }

// a < b
NSW6_FP_HD bool fp_lt(double a, double b) {
  const long long ia = fp_bits(a), ib = fp_bits(b);
  const long long ma = ia & FP_ABS, mb = ib & FP_ABS;
  const bool ordered = (ma <= FP_INF) & (mb <= FP_INF);
  const bool zeros = (ma | mb) == 0;
  return ordered & !zeros & (fp_key(ia) < fp_key(ib));
}

// a <= b
NSW6_FP_HD bool fp_le(double a, double b) {
  const long long ia = fp_bits(a), ib = fp_bits(b);
  const long long ma = ia & FP_ABS, mb = ib & FP_ABS;
  const bool ordered = (ma <= FP_INF) & (mb <= FP_INF);
  const bool zeros = (ma | mb) == 0;
  return ordered & (zeros | (fp_key(ia) <= fp_key(ib)));
}

NSW6_FP_HD bool fp_gt(double a, double b) { return fp_lt(b, a); }
NSW6_FP_HD bool fp_ge(double a, double b) { return fp_le(b, a); }

// |x| < c for a constant c > 0 (NaN: false)
NSW6_FP_HD bool fp_abs_lt(double x, double c) { return (fp_bits(x) & FP_ABS) < fp_bits(c); }

// x < c for a constant c > 0: every negative x and -0 below it, a positive x
// by its bits (NaN: false)
NSW6_FP_HD bool fp_lt_pos(double x, double c) {
  const long long b = fp_bits(x);
  return ((b & FP_ABS) <= FP_INF) & (b < fp_bits(c));
}

// max(x, c) as Kokkos::max, (x < c) ? c : x, for a constant c > 0
NSW6_FP_HD double fp_max_pos(double x, double c) { return fp_lt_pos(x, c) ? c : x; }

// x == 0 (either zero), by words: the 64-bit form ((bits & FP_ABS) == 0) was 92
// FP64-pipe instructions a cell of the column kernel
NSW6_FP_HD bool fp_is_zero(double x) { return ((fp_hi(x) << 1) | fp_lo(x)) == 0u; }

// x is +-inf or NaN (x * 0 != 0)
NSW6_FP_HD bool fp_not_finite(double x) { return (fp_hi(x) & 0x7FF00000u) == 0x7FF00000u; }

// x is NaN
NSW6_FP_HD bool is_nan_bits(double x) {
  const unsigned hi = fp_hi(x) & 0x7FFFFFFFu;
  return hi > 0x7FF00000u || (hi == 0x7FF00000u && fp_lo(x) != 0u);
}

// x is a positive normal number (not zero, subnormal, infinite or NaN)
NSW6_FP_HD bool fp_pos_normal(double x) {
  const long long b = fp_bits(x);
  return (b >= 0x0010000000000000ll) & (b < FP_INF);
}

// ---- comparisons with constants and the min / max they select (the cell
// physics' thresholds, clamps and limiters).  c: a positive normal constant
// (lt_negc: a negative one).  Each returns what the IEEE comparison (and the
// Kokkos::min / max select, (b < a) ? b : a and (a < b) ? b : a) returns.

NSW6_FP_HD double fp_from_bits(long long b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(b);
#else
  double x;
  std::memcpy(&x, &b, sizeof x);
  return x;
#endif
}

constexpr long long FP_SIGN = -0x7FFFFFFFFFFFFFFFll - 1;   // the sign bit; -0

NSW6_FP_HD bool is_one(double x) { return fp_bits(x) == 0x3FF0000000000000ll; }        // x == 1
NSW6_FP_HD bool is_nonneg(double x) {                                                    // x >= 0
  const long long b = fp_bits(x);
  return (b >= 0 && b <= FP_INF) || b == FP_SIGN;
}
NSW6_FP_HD bool is_finite_nonneg(double x) {                                             // 0 <= x < inf
  const long long b = fp_bits(x);
  return (unsigned long long)b < (unsigned long long)FP_INF || b == FP_SIGN;
}
NSW6_FP_HD bool is_zero(double x) { return fp_is_zero(x); }                              // x == 0
NSW6_FP_HD bool lt_z(double x) {                                                         // x < 0
  return (unsigned long long)fp_bits(x) - 0x8000000000000001ull < 0x7FF0000000000000ull;
}
NSW6_FP_HD bool gt_z(double x) {                                                         // x > 0
  const long long b = fp_bits(x);
  return b > 0 && b <= FP_INF;
}
NSW6_FP_HD bool ge_c(double x, double c) {                                               // x >= c
  const long long b = fp_bits(x);
  return b >= fp_bits(c) && b <= FP_INF;
}
NSW6_FP_HD bool gt_c(double x, double c) {                                               // x > c
  const long long b = fp_bits(x);
  return b > fp_bits(c) && b <= FP_INF;
}
NSW6_FP_HD bool le_c(double x, double c) {                                               // x <= c
  const long long b = fp_bits(x);
  return b <= fp_bits(c) && (b & FP_ABS) <= FP_INF;
}
NSW6_FP_HD bool lt_c(double x, double c) { return fp_lt_pos(x, c); }                     // x < c
NSW6_FP_HD bool lt_negc(double x, double c) {                                            // x < c, c < 0
  const long long b = fp_bits(x), m = b & FP_ABS;
  return b < 0 && m > (fp_bits(c) & FP_ABS) && m <= FP_INF;
}
NSW6_FP_HD double maxz(double x) { return lt_z(x) ? 0.0 : x; }                          // max(x, 0)
NSW6_FP_HD double maxc(double x, double c) { return fp_lt_pos(x, c) ? c : x; }          // max(x, c)
NSW6_FP_HD double minc(double x, double c) { return gt_c(x, c) ? c : x; }               // min(x, c)

// The limiters' d = max(q, 0) / dt (dt > 0, which the API enforces) is not
// negative: +-0, positive, +inf or NaN.  d < p exactly when p is positive and
// not NaN and d's magnitude bits are below p's; a < -d exactly when a is
// negative, not NaN and of larger magnitude.
NSW6_FP_HD bool lt_nn(double d, double p) {                                             // d < p
  const long long bp = fp_bits(p);
  return bp > 0 && bp <= FP_INF && (fp_bits(d) & FP_ABS) < bp;
}
NSW6_FP_HD double min_nn(double p, double d) { return lt_nn(d, p) ? d : p; }            // min(p, d)
NSW6_FP_HD bool lt_nd(double a, double d) {                                             // a < -d
  const long long ba = fp_bits(a), ma = ba & FP_ABS;
  return ba < 0 && ma > (fp_bits(d) & FP_ABS) && ma <= FP_INF;
}
NSW6_FP_HD double max_nd(double a, double d) {                                          // max(a, -d)
  return lt_nd(a, d) ? fp_of_words(fp_hi(d) ^ 0x80000000u, fp_lo(d)) : a;
}

// x + 0.0: -0 becomes +0, every other value stays (a NaN keeps its payload,
// where an FP64 addition gives the canonical NaN)
NSW6_FP_HD double plus_zero(double x) { return fp_bits(x) == FP_SIGN ? 0.0 : x; }

// Keys in the order of the doubles.  cmp_key: for non-NaN a and b, a >= b
// exactly when cmp_key(a) >= cmp_key(b), with -0 and +0 equal.
NSW6_FP_HD long long cmp_key(double x) {
  long long b = fp_bits(x);
  if (b == FP_SIGN) b = 0;
  return b < 0 ? (b ^ FP_ABS) : b;
}
// Order-preserving map double -> uint64 (total order, -0 < +0), used for exact
// atomic max/min of the per-level departure-distance extrema, and back.  By
// words: the 64-bit form's OR and NOT with the sign were two FP64-pipe
// instructions a row of the departure kernel.
NSW6_FP_HD unsigned long long order_key(double v) {
  const unsigned hi = fp_hi(v), lo = fp_lo(v);
  const unsigned neg = (unsigned)((int)hi >> 31);   // all ones for a negative number
  return ((unsigned long long)(hi ^ (neg | 0x80000000u)) << 32) | (lo ^ neg);
}
NSW6_FP_HD double key_value(unsigned long long k) {
  return fp_from_bits((long long)((k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k));
}

}  // namespace nsw6
