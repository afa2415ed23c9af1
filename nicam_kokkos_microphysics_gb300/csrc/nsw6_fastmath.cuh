// Transcendental functions of the NSW6 kernels as policies.
//
// FastMath, the production policy, evaluates exp, log and pow in 64-bit fixed
// point on the integer pipe (nsw6_soft.cuh): on GB300 an FP64 instruction
// takes 16 to 19 cycles of an SM, an integer one about half a cycle, and exp,
// log and pow took 9, 17 and 28 FP64 instructions (a table-driven evaluation
// in doubles, which these replaced) where they take some 65, 85 and 110 integer
// ones.  pow(x, y) is 2^(y log2 x) with log2 x and the product in fixed point,
// so nothing is rounded before the result.  Errors against 128-bit references
// (10^6 arguments each): exp at most 0.518 units in the last place, 99.8 %
// correctly rounded; log 0.52, 99.99 %; pow 0.52, 99.7 %.  The evaluation in
// doubles had 96 %, 95 % and 2 units for pow.  One 16900 x 42 region, FP64:
// step 2.134 -> 1.944 ms.
//
// The tables (7 KB) are built on the host in extended precision.  The cell and
// derivative kernels stage them in shared memory; the column and saturation
// kernels, few of whose cells ask for them, read them through L1.
#pragma once

#include <cstdint>

#include "nsw6_fpcmp.cuh"
#include "nsw6_soft.cuh"

namespace nsw6 {

// Table layout, in doubles: T[256], LT[512] (64-bit numbers), IC[512] (16-bit).
constexpr int FM_TABLE_DOUBLES = SOFT_EXP_N + SOFT_LOG_N + SOFT_LOG_N / 4;

struct FastMath {
  SoftTables T;
  __device__ __forceinline__ explicit FastMath(const double* tab)
      : T{reinterpret_cast<const u64*>(tab), reinterpret_cast<const u64*>(tab + SOFT_EXP_N),
          reinterpret_cast<const unsigned short*>(tab + SOFT_EXP_N + SOFT_LOG_N)} {}

  __device__ __forceinline__ double exp(double x) const { return soft_exp(x, T); }

  __device__ __forceinline__ double log(double x) const {
    const long long bits = __double_as_longlong(x);
    // x normal and finite, positive (the signed bits order the positive doubles)
    if (!(bits >= 0x0010000000000000ll && bits < 0x7FEFFFFFFFFFFFFFll)) return soft_slow_log(x);
    // |x - 1| < 2^-7 (x - 1 is exact there, Sterbenz): the fixed point's
    // absolute error would show
    if (bits > 0x3FEFC00000000000ll && bits < 0x3FF0200000000000ll) return log1p_near1(x - 1.0);
    return soft_log((u64)bits, T);
  }

  // log1p(f) = f + f^2 (-1/2 + f (1/3 + ... + f (-1/8))), whose truncation
  // error is below 2e-18 relative for |f| < 1/128.
  __device__ __forceinline__ static double log1p_near1(double f) {
    double q = __fma_rn(f, -1.2500000000000000e-01, 1.4285714285714285e-01);
    q = __fma_rn(q, f, -1.6666666666666666e-01);
    q = __fma_rn(q, f, 2.0e-01);
    q = __fma_rn(q, f, -0.25);
    q = __fma_rn(q, f, 3.3333333333333331e-01);
    q = __fma_rn(q, f, -0.5);
    return __fma_rn(q, __dmul_rn(f, f), f);
  }

  // x^y for x >= 0 (the only use here); x == 0 gives 0 for y > 0.
  __device__ __forceinline__ double pow(double x, double y) const {
    if (fp_is_zero(x)) return fp_gt(y, 0.0) ? 0.0 : soft_slow_pow(x, y);
    return soft_pow(x, y, T);
  }
};

// FP32 transcendentals of the mixed-precision path (CUDA's expf / logf /
// powf, within 2 ulp of FP32).
struct FloatMath {
  __device__ __forceinline__ float exp(float x) const { return ::expf(x); }
  __device__ __forceinline__ float log(float x) const { return ::logf(x); }
  __device__ __forceinline__ float pow(float x, float y) const { return ::powf(x, y); }
};

// Same interface on top of the CUDA math library (used to separate the
// effects of the fast transcendentals from everything else).
struct LibMath {
  __device__ __forceinline__ double exp(double x) const { return ::exp(x); }
  __device__ __forceinline__ double log(double x) const { return ::log(x); }
  __device__ __forceinline__ double pow(double x, double y) const { return ::pow(x, y); }
};

}  // namespace nsw6
