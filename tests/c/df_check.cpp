// Host check of the double-float quotient (ffv_df.cuh) over the range that its header states: its
// error against the quotient in extended precision, and special divisors, both beside the plain form
// with two divisions.  Prints the number of failures and exits nonzero if there is any.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>

#define __host__
#define __device__
#define __forceinline__ inline
#define __noinline__
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static inline float __fdiv_rn(float a, float b) { return a / b; }
static inline float __frcp_rn(float a) { return 1.0f / a; }
using std::isnan;
#include "ffv_df.cuh"

static uint64_t state = 0x9E3779B97F4A7C15ull;
static uint64_t next_u64() {
  state ^= state << 13;
  state ^= state >> 7;
  state ^= state << 17;
  return state;
}
// a pair of exponent e, mantissas and the gap to the low part random
static df pair(int e) {
  const float hi = std::ldexp((float)((next_u64() & 0x7FFFFF) | 0x800000), e - 23);
  const float lo = std::ldexp((float)(int64_t)(next_u64() & 0xFFFFFF) - 8388608.0f, e - 23 - 25);
  const df p = fast_two_sum(next_u64() & 1 ? hi : -hi, lo);
  return p;
}

// the plain form
static df div_plain(df x, df y) {
  const float q1 = __fdiv_rn(x.hi, y.hi);
  const df r = df_sub(x, df_mul_f(y, q1));
  return fast_two_sum(q1, __fdiv_rn(r.hi, y.hi));
}

int main() {
  long bad = 0, checked = 0;
  double worst = 0.0;
  // divisors over the whole normal range, quotients and dividends where the low parts are normal too
  for (int ey = -126; ey <= 127; ey++)
    for (int ex = -70; ex <= 126; ex++) {
      if (ex - ey < -70 || ex - ey > 126) continue;
      for (int i = 0; i < 40; i++) {
        const df x = pair(ex), y = pair(ey), q = df_div(x, y);
        if (std::isinf((double)x.hi) || std::isinf((double)y.hi)) continue;
        const long double want = ((long double)x.hi + x.lo) / ((long double)y.hi + y.lo);
        if (std::fabs(want) > 3.0e38L) continue;
        const double err = (double)(std::fabs(((long double)q.hi + q.lo - want) / want));
        checked++;
        if (err > worst) worst = err;
        // df_mul_f, df_sub (2^-46 of the larger operand, a quotient) and the second quotient's rounding
        if (!(err <= std::ldexp(1.0, -44)) && bad++ < 10)
          std::printf("%a / %a: error %g, plain %g\n", (double)x.hi, (double)y.hi, err,
                      (double)(std::fabs(((long double)div_plain(x, y).hi + div_plain(x, y).lo - want) / want)));
      }
    }
  // special operands: as the plain form
  const float ends[] = {0.0f, -0.0f, 1.0f, -2.5f, INFINITY, -INFINITY, NAN};
  for (float a : ends)
    for (float y : ends) {
      const df got = df_div(df_make(a), df_make(y)), want = div_plain(df_make(a), df_make(y));
      checked++;
      if (!(isnan(got.hi) == isnan(want.hi) && (isnan(want.hi) || got.hi == want.hi)) && bad++ < 10)
        std::printf("%a / %a: %a, not %a\n", (double)a, (double)y, (double)got.hi, (double)want.hi);
    }
  // single quotients: as the division, whatever the operands
  const float special[] = {0.0f, -0.0f, 1.0f, -3.0f, 1e-45f, -1e-40f, 1.2e-38f, 2.3e-38f, 1e-20f, 1e20f, 4.2e37f,
                           8.6e37f, -1.7e38f, 3.4e38f, INFINITY, -INFINITY, NAN};
  const auto single = [&](float a, float y) {
    const float got = quotient(a, y, __frcp_rn(y)), want = a / y;
    checked++;
    if (!(got == want || (isnan(got) && isnan(want))) && bad++ < 20)
      std::printf("quotient %a / %a: %a, not %a\n", (double)a, (double)y, (double)got, (double)want);
  };
  for (float a : special)
    for (float y : special) single(a, y);
  for (int i = 0; i < 4000000; i++) {
    uint32_t u = (uint32_t)next_u64(), v = (uint32_t)next_u64();
    float a, y;
    memcpy(&a, &u, 4);
    memcpy(&y, &v, 4);
    single(a, y);
  }
  for (int i = 0; i < 4000000; i++) single(pair((int)(next_u64() % 40) - 20).hi, pair((int)(next_u64() % 40) - 20).hi);
  std::printf("%ld checked, largest error of a double-float quotient %.3g, %ld failures\n", checked, worst, bad);
  return bad != 0;
}
