// The integer-pipe arithmetic of nsw6_soft.cuh on the host: quotients, roots
// and conversions against the host's IEEE operations bit for bit, exp, log and
// pow against long double.  Prints the counts and largest errors.
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "nsw6_soft.cuh"

using namespace nsw6;

static u64 bits(double x) {
  u64 b;
  std::memcpy(&b, &x, 8);
  return b;
}
static bool same(double a, double b) { return bits(a) == bits(b) || (a != a && b != b); }
static bool same(float a, float b) { return std::memcmp(&a, &b, 4) == 0 || (a != a && b != b); }
static double ulps(double got, long double want) {
  int e;
  std::frexp((double)want, &e);
  return (double)(std::fabs((long double)got - want) / std::ldexp(1.0L, e - 53));
}

int main() {
  std::vector<u64> t(SOFT_EXP_N), lt(SOFT_LOG_N);
  std::vector<unsigned short> ic(SOFT_LOG_N);
  for (int j = 0; j < SOFT_EXP_N; ++j) t[j] = (u64)(exp2l((long double)j / SOFT_EXP_N) * 9223372036854775808.0L + 0.5L);
  for (int j = 0; j < SOFT_LOG_N; ++j) {
    const int lo = SOFT_LOG_N + j, n = (32768 * SOFT_LOG_N + lo - 1) / lo;
    ic[j] = (unsigned short)n;
    lt[j] = (u64)(-log2l((long double)n / 32768.0L) * 18446744073709551616.0L + 0.5L);
  }
  const SoftTables T{t.data(), lt.data(), ic.data()};
  std::mt19937_64 g(7);
  // mantissas at random, with long runs of zeros or ones, and next to powers of two
  auto number = [&](int spread) {
    u64 m = g();
    switch (g() % 4) {
      case 0: m &= ~((1ull << (g() % 52)) - 1); break;
      case 1: m |= (1ull << (g() % 52)) - 1; break;
      default: break;
    }
    const u64 b = (m & SOFT_MANT) | ((u64)(1023 - spread + (int)(g() % (2 * spread))) << 52) | (g() & (1ull << 63));
    double x;
    std::memcpy(&x, &b, 8);
    return x;
  };
  long bad_div = 0, bad_rcp = 0, bad_sqrt = 0, bad_cvt = 0;
  for (int i = 0; i < 4000000; ++i) {
    const double b = number(i % 3 == 0 ? 1020 : 120);
    double a = number(i % 3 == 0 ? 1020 : 120);
    if (i % 7 == 0) a = b * (1.0 + ((int)(g() % 9) - 4) * 2.3e-16);   // quotients next to 1
    if (i % 11 == 0) a = (float)a * (double)(float)b;                  // exact quotients
    if (i % 13 == 0) a = i % 2 ? 0.0 : -0.0;
    bad_div += !same(soft_div(a, b), a / b);
    const double rb = 1.0 / b, q = a * rb, m = std::fma(std::fma(-q, b, a), rb, q);
    // div_rn is Markstein's form, the correctly rounded quotient where that is normal
    if (std::fabs(a) > 1e-140 && std::fabs(a) < 1e140 && std::fabs(b) > 1e-140 && std::fabs(b) < 1e140)
      bad_div += !same(soft_div_rn(a, soft_divisor(b), b), a / b);
    else if (a == 0.0 && std::isnormal(rb))
      bad_div += !same(soft_div_rn(a, soft_divisor(b), b), m);
    bad_rcp += !same(soft_rcp(soft_divisor(b), b), rb);
    double x = std::fabs(a);
    if (i % 5 == 0) {   // squares and their neighbours
      const double s = (float)x;
      x = i % 2 ? s * s : std::nextafter(s * s, i % 4 ? 1e300 : 0.0);
    }
    bad_sqrt += !same(soft_sqrt(x), std::sqrt(x));
    bad_cvt += !same(soft_d2f(a), (float)a) + !same(soft_f2d((float)b), (double)(float)b);
  }
  const double special[] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 5e-324, -5e-324, 1e-310, 2.2250738585072014e-308,
                            1.7976931348623157e308, 1.0, -1.0, 2.0, 0.5, 3.0, 1e-300, 1e300, 1.1754943508222875e-38,
                            1.17549429e-38, 3.4028235677973366e38, 3.4028234e38, 1e-45, 1e-39, 1.7014118346046923e38,
                            4.0, 3.9999999999999996, 1.9999999999999998, 1.0000000000000002, 0.99999999999999989};
  for (double a : special) {
    for (double b : special) bad_div += !same(soft_div(a, b), a / b);
    bad_sqrt += !same(soft_sqrt(a), std::sqrt(a));
    bad_cvt += !same(soft_d2f(a), (float)a) + !same(soft_f2d((float)a), (double)(float)a);
  }
  auto unit = [&] { return (double)(g() >> 11) * 0x1p-53; };
  double e_exp = 0.0, e_log = 0.0, e_pow = 0.0;
  const double powers[] = {2.47, 1.15, 0.75, 0.33333333, 1.33, -1.79, 0.16};
  for (int i = 0; i < 300000; ++i) {
    double x = (unit() - 0.5) * (i % 3 == 0 ? 1400 : i % 3 == 1 ? 80 : 2);
    if (i % 97 == 0) x *= 1e-10;
    e_exp = std::fmax(e_exp, ulps(soft_exp(x, T), expl(x)));
    x = std::exp((unit() - 0.5) * (i % 3 ? 100 : 1200));
    if (std::fabs(x - 1.0) < 0.0078125) x += 0.02;
    e_log = std::fmax(e_log, ulps(soft_log(bits(x), T), logl(x)));
    const double y = i % 2 ? powers[g() % 7] : (unit() - 0.5) * 6;
    x = i % 10 == 0 ? 1.0 + (unit() - 0.5) * 0.01 : std::exp((unit() - 0.7) * 60);
    e_pow = std::fmax(e_pow, ulps(soft_pow(x, y, T), powl(x, y)));
  }
  long bad_edge = 0;
  for (double x : {0.0, -0.0, 5e-324, 1e-17, -1e-17, -1e-16, 707.9, -707.9, 710.0, -746.0, (double)INFINITY, (double)-INFINITY})
    bad_edge += !(std::fabs(soft_exp(x, T) - std::exp(x)) <= 1.2e-16 * std::exp(x)) && soft_exp(x, T) != std::exp(x);
  for (double x : {1.0, 2.0, 0.25, 0.99999999999999989, 1.0000000000000002, 5e-324, 1e300})
    for (double y : {2.47, -1.79, 64.0, 100.0, 1e-9, -1e-9, 1e-20, 300.0, 0.0})
      bad_edge += !(std::fabs(soft_pow(x, y, T) - std::pow(x, y)) <= 2.3e-16 * std::pow(x, y)) &&
                  soft_pow(x, y, T) != std::pow(x, y);
  std::printf("div %ld rcp %ld sqrt %ld cvt %ld edge %ld exp %.3f log %.3f pow %.3f\n", bad_div, bad_rcp, bad_sqrt,
              bad_cvt, bad_edge, e_exp, e_log, e_pow);
  return 0;
}
