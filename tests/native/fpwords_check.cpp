// The forms of nsw6_fpcmp.cuh that go by the two words of a double, as both
// targets compile them, against the IEEE operations: special values pairwise,
// random bit patterns and near pairs, and patterns with one word all zeros or
// ones.  Prints the number of mismatches.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <vector>

#include "nsw6_fpcmp.cuh"

using namespace nsw6;

static double from_bits(unsigned long long b) {
  double x;
  std::memcpy(&x, &b, sizeof x);
  return x;
}
static unsigned long long bits(double x) {
  unsigned long long b;
  std::memcpy(&b, &x, sizeof b);
  return b;
}
static bool same(double x, double y) { return bits(x) == bits(y) || (std::isnan(x) && std::isnan(y)); }

static long long check(double a, double b) {
  long long bad = 0;
  bad += bits(fp_of_words(fp_hi(a), fp_lo(a))) != bits(a);
  bad += fp_is_zero(a) != (a == 0.0);
  bad += fp_not_finite(a) != !std::isfinite(a);
  bad += is_nan_bits(a) != std::isnan(a);
  bad += is_finite_nonneg(a) != (a >= 0.0 && std::isfinite(a));
  bad += fp_pos_normal(a) != (a > 0.0 && std::isnormal(a));
  const double d = std::fabs(b);
  bad += !same(max_nd(a, d), (a < -d) ? -d : a);
  bad += bits(key_value(order_key(a))) != bits(a);
  if (!std::isnan(a) && !std::isnan(b)) {
    bad += (cmp_key(a) >= cmp_key(b)) != (a >= b);
    // -0 below +0
    const bool below = a < b || (a == b && std::signbit(a) && !std::signbit(b));
    bad += (order_key(a) < order_key(b)) != below;
  }
  return bad;
}

int main() {
  const double inf = std::numeric_limits<double>::infinity();
  std::vector<double> sp = {0.0, -0.0, 1.0, -1.0, 4.9e-324, -4.9e-324, 2.2250738585072014e-308,
                            -2.2250738585072014e-308, 1.7976931348623157e308, -1.7976931348623157e308, inf, -inf,
                            from_bits(0x7FF0000000000001ull), from_bits(0xFFF0000000000001ull),
                            from_bits(0x7FF8000000000000ull), from_bits(0xFFFFFFFFFFFFFFFFull)};
  // one word at an edge, the other anything
  for (unsigned long long w : {0x00000000ull, 0x00000001ull, 0x7FEFFFFFull, 0x7FF00000ull, 0x7FF00001ull, 0x80000000ull,
                               0x80000001ull, 0xFFF00000ull, 0xFFFFFFFFull})
    for (unsigned long long v : {0x00000000ull, 0x00000001ull, 0x7FFFFFFFull, 0x80000000ull, 0xFFFFFFFFull})
      sp.push_back(from_bits((w << 32) | v));
  long long bad = 0;
  for (double a : sp)
    for (double b : sp) bad += check(a, b);
  std::mt19937_64 rng(99);
  for (int i = 0; i < 2000000; ++i) {
    const unsigned long long r = rng();
    bad += check(from_bits(r), from_bits(rng()));
    bad += check(from_bits(r), from_bits(r + rng() % 5 - 2));
    bad += check(from_bits(r & 0xFFFFFFFF00000000ull), from_bits(r & 0xFFFFFFFFull));
  }
  std::printf("mismatches %lld\n", bad);
  return bad == 0 ? 0 : 1;
}
