// Host check of the bit-level FP64 helpers (ffv_fp64.cuh) against the plain expressions they
// stand for: random bit patterns over the whole exponent range, random pairs of moderate size,
// quotients near rounding midpoints, zeros, subnormals, infinities and NaN.  Prints the number of
// mismatches and exits nonzero if there is any.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>

#include "ffv_fp64.cuh"

static uint64_t state = 0x9E3779B97F4A7C15ull;
static uint64_t next_u64() {
  state ^= state << 13;
  state ^= state >> 7;
  state ^= state << 17;
  return state;
}
static double dbl(uint64_t u) { return f64::of_bits(u); }
// mantissa random, exponent within +-span of 1
static double around_one(int span) {
  const uint64_t e = 1023 - span + next_u64() % (2 * span + 1);
  return dbl((next_u64() & 0x800fffffffffffffull) | (e << 52));
}
static bool same(double a, double b) {
  return (std::isnan(a) && std::isnan(b)) || f64::bits(a) == f64::bits(b);
}

static long bad = 0, checked = 0;
static void expect(bool ok, const char *what, double x, double y) {
  checked++;
  if (!ok && bad++ < 10) std::printf("%s: %a %a\n", what, x, y);
}

static void one(double x) {
  expect(f64::is_nan(x) == std::isnan(x), "is_nan", x, 0);
  expect(f64::ge0(x) == (x >= 0.0), "ge0", x, 0);
  expect(f64::le0(x) == (x <= 0.0), "le0", x, 0);
  expect(f64::gt0(x) == (x > 0.0), "gt0", x, 0);
  expect(f64::lt0(x) == (x < 0.0), "lt0", x, 0);
  expect(same(f64::neg(x), -x), "neg", x, 0);
}

static void two(double x, double y) {
  if (!std::isnan(y)) expect(f64::abs_gt(x, y) == (std::fabs(x) > std::fabs(y)), "abs_gt", x, y);
  if (!std::isnan(y) && y != 0.0) {
    expect(f64::lt(x, y) == (x < y), "lt", x, y);
    expect(f64::le(x, y) == (x <= y), "le", x, y);
    expect(f64::gt(x, y) == (x > y), "gt", x, y);
    expect(f64::ge(x, y) == (x >= y), "ge", x, y);
  }
  expect(same(f64::div(x, f64::rcp(y)), x / y), "div", x, y);
}

// the reference's limiter on the two faces of an axis (m0_deltavalues.c:23-57,
// m0_reconctruct.c:160-207)
static double face(double df, double db, double h) {
  double grad = 0.0;
  if (std::fabs(df) > 1e-10) {
    const double product = (-db / h) * (df / h);
    if (product > 0.0) grad = std::fabs(db / h) > std::fabs(df / h) ? df / h : -db / h;
  }
  return (0.5 * h) * grad;
}
static void limiter(double dp, double dm) {
  for (int k : {-12, -3, 0}) {
    const double h = std::ldexp(1.0, k);
    double cp, cm;
    f64::minmod_pair(dp, dm, 1.0 / h, cp, cm);
    expect(same(cp, face(dp, dm, h)), "minmod +", dp, dm);
    expect(same(cm, face(dm, dp, h)), "minmod -", dp, dm);
  }
}

int main() {
  const double inf = INFINITY, nan = NAN;
  const double special[] = {0.0, -0.0, 1.0, -1.0, 1e-10, -1e-10, 1.0000000000000002e-10, 9.999999999999999e-11,
                            4.9e-324, -4.9e-324, 2.2250738585072014e-308, -2.3e-308, 1e-300, -1e-290, 1e-160,
                            -3e-165, 1.7976931348623157e308, -1e308, inf, -inf, nan, 3.0, 2.0 / 3.0, 1e200, 1e-200};
  for (double x : special) {
    one(x);
    for (double y : special) {
      two(x, y);
      limiter(x, y);
    }
    for (int i = 0; i < 2000; i++) {
      const double y = around_one(30);
      two(x, y);
      two(y, x);
      limiter(x, y);
      limiter(y, x);
    }
  }
  for (int i = 0; i < 4000000; i++) {
    const double x = dbl(next_u64()), y = dbl(next_u64());
    one(x);
    two(x, y);
    const double a = around_one(40), b = around_one(40);
    two(a, b);
    // a quotient just beside a midpoint between two doubles: a = b (m + half an ulp), rounded
    const double m = around_one(0);
    two(std::fma(b, m, b * std::ldexp(m > 0 ? 1.0 : -1.0, -53)), b);
    two(a, std::nextafter(std::ldexp(1.0, i % 60 - 30), i & 1 ? 0.0 : 1e300));  // divisors beside powers of two
    limiter(a, around_one(60));
    limiter(a, f64::neg(a));
  }
  std::printf("%ld checks, %ld mismatches\n", checked, bad);
  return bad != 0;
}
