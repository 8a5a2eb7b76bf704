// Division by a value whose reciprocal is kept.
#pragma once
#include <cfloat>
#include <cmath>

#ifdef __CUDACC__
#define LBMB_HD __host__ __device__ __forceinline__
#else
#define LBMB_HD inline
#endif

namespace lbmb {

// The reciprocal that quotient() takes for b: 1 / b, the largest finite value
// where that overflows.
LBMB_HD double reciprocal(double b) {
  const double y = 1.0 / b;
  return y > DBL_MAX ? DBL_MAX : y;
}

// a / b rounded to nearest, from y = reciprocal(b) and with no division on
// the way (Markstein 1990: from a quotient within an ulp, its exact remainder
// and y, one correction rounds correctly; the first correction here brings the
// product a y within an ulp). Infinite and NaN operands and quotients that
// overflow give what the division gives; next to underflow the remainder is
// inexact and the result may be off in the last place.
LBMB_HD double quotient(double a, double b, double y) {
  const double q = a * y;
  const double r = std::fma(-q, b, a);
  const double q1 = std::fma(r, y, q);
  const double q2 = std::fma(std::fma(-q1, b, a), y, q1);
  return std::fabs(r) <= DBL_MAX ? q2 : q;
}

}  // namespace lbmb
