// dv_div.h -- x / d for a divisor that stays the same over many x, in host and
// device code.
//
// With y = 1 / d rounded to nearest, q0 = x y is within two units in the last
// place of x / d, q1 = q0 + (x - q0 d) y is within one, and
// q2 = q1 + (x - q1 d) y is x / d rounded to nearest (P. Markstein, IBM J. Res.
// Dev. 34 (1990), 111-119, theorem on the last step of a division: q1 a faithful
// quotient, y the rounded reciprocal, the remainder exact by a fused
// multiply-add).  Five dependent operations and no branch on the way, where the
// compiler's division has to form the reciprocal first.  The theorem wants
// remainders and quotients away from underflow and overflow: other x (zeros,
// infinities and NaN among them) take the ordinary division, and so does
// every x when d is not in [1, kDivMost].
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define DV_HD __host__ __device__
#else
#define DV_HD
#endif

namespace dv {

template <class R> struct DivRange;
// |x| between these, and 1 <= d <= kMost, keep x, q and x - q d normal
template <> struct DivRange<double> {
  static constexpr double kLeast = 1e-200, kLargest = 1e300, kMost = 1e60;
};
template <> struct DivRange<float> {
  static constexpr float kLeast = 1e-20f, kLargest = 1e37f, kMost = 1e6f;
};

DV_HD inline double dv_fma(double a, double b, double c) { return fma(a, b, c); }
DV_HD inline float dv_fma(float a, float b, float c) { return fmaf(a, b, c); }

// The reciprocal that div_by takes; NaN sends every x to the ordinary division.
template <class R>
DV_HD inline R div_reciprocal(R d) {
  return (d >= R(1) && d <= DivRange<R>::kMost) ? R(1) / d : R(NAN);
}

template <class R>
DV_HD inline R div_by(R x, R d, R y) {
  const R a = x < R(0) ? -x : x;
  if (a >= DivRange<R>::kLeast && a <= DivRange<R>::kLargest && y == y) {
    R q = x * y;
    q = dv_fma(dv_fma(-q, d, x), y, q);
    return dv_fma(dv_fma(-q, d, x), y, q);
  }
  return x / d;
}

}  // namespace dv
