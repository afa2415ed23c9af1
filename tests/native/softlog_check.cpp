// The fixed-point exp, log and pow of nsw6_soft.cuh on the host against long
// double where their last steps can go wrong: results next to a power of two,
// whose rounding carries into the exponent, and arguments at the edges of the
// tables' intervals.  Prints the largest errors in units in the last place.
#include <cstdio>
#include <cstring>
#include <vector>

#include "nsw6_soft.cuh"

using namespace nsw6;

static u64 bits(double x) {
  u64 b;
  std::memcpy(&b, &x, 8);
  return b;
}
static double near(double x, int ulps) {   // x moved by that many units in the last place
  const u64 b = bits(x) + (u64)(long long)ulps;
  double y;
  std::memcpy(&y, &b, 8);
  return y;
}
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
  double e_log = 0.0, e_exp = 0.0, e_pow = 0.0;
  auto check_log = [&](double x) {
    if (std::fabs(x - 1.0) >= 0.0078125) e_log = std::fmax(e_log, ulps(soft_log(bits(x), T), logl(x)));
  };
  // logarithms next to +-2^e: the doubles around exp(+-2^e)
  for (int s = -1; s <= 1; s += 2)
    for (int e = -6; e <= 9; ++e)
      for (int i = -600; i <= 600; ++i) check_log(near((double)expl(s * std::ldexp(1.0L, e)), i));
  // the edges of the logarithm's intervals and of its exponents
  for (int e = -1022; e < 1023; e += e > -40 && e < 40 ? 1 : 37)
    for (int j = 0; j <= SOFT_LOG_N; ++j)
      for (int i = -2; i <= 2; ++i) {
        const double x = near(std::ldexp(1.0 + (double)j / SOFT_LOG_N, e), i);
        if (x >= 2.2250738585072014e-308) check_log(x);
      }
  // exponentials at the edges of the table's intervals (next to powers of two at every 256th)
  for (int k = -1000 * SOFT_EXP_N; k <= 1000 * SOFT_EXP_N; k += k > -4096 && k < 4096 ? 1 : 61)
    for (int i = -3; i <= 3; ++i) {
      const double x = k ? near((double)(k * (logl(2.0L) / SOFT_EXP_N)), i) : i * 1.0e-17;
      e_exp = std::fmax(e_exp, ulps(soft_exp(x, T), expl(x)));
    }
  // powers next to powers of two
  for (double y : {2.47, 1.15, 0.75, 0.33333333, 1.33, -1.79, 0.16, 2.0, -3.0, 0.5})
    for (int k = -60; k <= 60; ++k)
      for (int i = -20; i <= 20; ++i) {
        const double x = near((double)powl(2.0L, k / (long double)y), i);
        e_pow = std::fmax(e_pow, ulps(soft_pow(x, y, T), powl(x, y)));
      }
  std::printf("log %.3f exp %.3f pow %.3f\n", e_log, e_exp, e_pow);
  return 0;
}
