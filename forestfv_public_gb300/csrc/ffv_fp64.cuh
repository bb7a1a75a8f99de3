// FP64 arithmetic of the reference-exact kernels with fewer instructions on the FP64 pipe.
//
// GB300 issues one FP64 instruction per warp and SM sub-partition every 64 cycles (2 lanes per
// SM and clock); comparisons, min / max and conversions of doubles go through the same pipe, and
// a correctly rounded division is a sequence of about ten of them.  The reference-exact kernels
// are bound by that pipe (80-86 % busy, the issue slots 8 % busy), so whatever can be decided or
// scaled on the bit patterns is done with integer instructions here, and quotients by a common
// divisor share its reciprocal.  Every function returns the bits of the plain expression it
// stands for; a host test checks them (tests/test_fp64.py).
//
// Compiles for the host too.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#ifndef __CUDACC__
#define FFV_F64_FN static inline
#define FFV_F64_COLD static
#else
#define FFV_F64_FN __host__ __device__ __forceinline__
#define FFV_F64_COLD static __host__ __device__ __noinline__
#endif

namespace f64 {

constexpr uint64_t kSign = 0x8000000000000000ull, kInf = 0x7ff0000000000000ull;

FFV_F64_FN uint64_t bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
FFV_F64_FN double of_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}
FFV_F64_FN uint64_t abs_bits(double x) { return bits(x) & ~kSign; }
FFV_F64_FN double neg(double x) { return of_bits(bits(x) ^ kSign); }

FFV_F64_FN bool is_nan(double x) { return abs_bits(x) > kInf; }
// |x| > |y| for y not NaN (false where x is NaN)
FFV_F64_FN bool abs_gt(double x, double y) {
  const uint64_t a = abs_bits(x);
  return a > abs_bits(y) && a <= kInf;
}
// x >= 0, x <= 0 (both zeros count; false for NaN)
FFV_F64_FN bool ge0(double x) {
  const uint64_t u = bits(x);
  return u <= kInf || u == kSign;
}
FFV_F64_FN bool le0(double x) {
  const uint64_t u = bits(x);
  return (u >= kSign && u <= (kSign | kInf)) || u == 0;
}
FFV_F64_FN bool gt0(double x) { return bits(x) - 1 < kInf; }
FFV_F64_FN bool lt0(double x) {
  const uint64_t u = bits(x);
  return u > kSign && u <= (kSign | kInf);
}
// order-preserving integer of a double that is not NaN (-0 just below +0)
FFV_F64_FN int64_t order_key(double x) {
  const int64_t s = (int64_t)bits(x);
  return s ^ ((s >> 63) & 0x7fffffffffffffffll);
}
// x < y, x <= y, x > y, x >= y for a y that is neither NaN nor zero (false where x is NaN)
FFV_F64_FN bool lt(double x, double y) { return order_key(x) < order_key(y) && !is_nan(x); }
FFV_F64_FN bool le(double x, double y) { return order_key(x) <= order_key(y) && !is_nan(x); }
FFV_F64_FN bool gt(double x, double y) { return order_key(x) > order_key(y) && !is_nan(x); }
FFV_F64_FN bool ge(double x, double y) { return order_key(x) >= order_key(y) && !is_nan(x); }

// A divisor and its reciprocal, rounded to nearest.
struct Rcp {
  double d, r;
};
FFV_F64_FN Rcp rcp(double d) { return Rcp{d, 1.0 / d}; }

FFV_F64_COLD double div_plain(double x, double d) { return x / d; }

// 2^-400 <= |x| < 2^400
FFV_F64_FN bool moderate(double x) {
  return (((uint32_t)(bits(x) >> 32) & 0x7fffffffu) - (623u << 20)) < (800u << 20);
}

// x / d.  The quotient from the rounded reciprocal, corrected by its exact remainder -- the
// closing step of Markstein's division (P. Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", 1990; Brisebarre, Muller and Raina, "Accelerating
// correctly rounded floating-point division when the divisor is known in advance", 2004): three
// instructions per quotient where several share a divisor.  Operands outside the range where
// the remainder is exact (and infinities, NaN, a zero divisor) take the plain division.
FFV_F64_FN double div(double x, const Rcp &c) {
  const double q = x * c.r;
  if (moderate(x) && moderate(q)) return fma(fma(-q, c.d, x), c.r, q);
  if ((bits(x) & ~kSign) == 0 && moderate(c.d)) return q;  // a zero of the quotient's sign
  return div_plain(x, c.d);
}

// The limited face increments of one variable along one axis, between two neighbours of the
// cell's own level at spacing h, a power of two, the faces at h / 2: with the differences
// dp, dm to the two neighbours the reference's
//   (-dm / h) * (dp / h) > 0 ? (|dm / h| > |dp / h| ? dp / h : -dm / h) : 0, where |dp| > 1e-10,
// times h / 2 for the first face, and the same with the roles exchanged for the second.  The
// scalings by powers of two are exact, so signs and magnitudes decide on the bit patterns and
// the increments are half the smaller difference.  Differences so small or large that a product
// or quotient leaves the normal range take the plain form (ih = 1 / h).
FFV_F64_COLD double minmod_plain(double df, double db, double ih) {
  const double sf = df * ih, sb = -db * ih;
  double grad = 0.0;
  if (fabs(df) > 1e-10 && sb * sf > 0.0) grad = fabs(sb) > fabs(sf) ? sf : sb;
  return (0.5 / ih) * grad;
}
FFV_F64_FN bool ordinary(uint64_t a) {  // 2^-500 <= |x| < 2^500, a = abs_bits(x)
  return a - (523ull << 52) < (1000ull << 52);
}
FFV_F64_FN void minmod_pair(double dp, double dm, double ih, double &cp, double &cm) {
  const uint64_t tiny = 0x3ddb7cdfd9d7bdbbull;  // 1e-10
  const uint64_t ap = abs_bits(dp), am = abs_bits(dm);
  cp = cm = 0.0;
  if (((bits(dp) ^ bits(dm)) >> 63) && ap - 1 < kInf && am - 1 < kInf) {
    if (ordinary(ap) && ordinary(am)) {
      // the halves, an exponent one lower; the increments point towards the first neighbour
      const uint64_t one = 1ull << 52;
      if (ap > tiny) cp = of_bits((am > ap ? bits(dp) : bits(dm) ^ kSign) - one);
      if (am > tiny) cm = of_bits((ap > am ? bits(dm) : bits(dp) ^ kSign) - one);
    } else {
      cp = minmod_plain(dp, dm, ih);
      cm = minmod_plain(dm, dp, ih);
    }
  }
}

}  // namespace f64
