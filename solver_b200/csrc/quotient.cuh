// The division of the advection's limiter, rounded as the division operator
// rounds it.  Host code can include this (the tests do).
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define OFB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define OFB_HOST_DEVICE inline
#endif

namespace ofb {

// n / d rounded to nearest, from an approximation r of 1 / d of relative error
// below 2^-19.  A step of Halley's cubic iteration (error 2^-57, and a rounding)
// leaves r within an ulp; 1 - d r is then exact and a Newton step rounds r
// correctly, but where the fraction of d is all ones; n r is within an ulp of the
// quotient, its residual is exact, and adding residual times r rounds correctly
// (Markstein, IBM J. Res. Dev. 34, 1990, theorems on the reciprocal and the
// quotient).
OFB_HOST_DEVICE double quotient_from(double n, double d, double r) {
  double e = fma(-d, r, 1.0);
  e = fma(e, e, e);
  r = fma(r, e, r);
  r = fma(r, fma(-d, r, 1.0), r);
  const double q = n * r;
  return fma(fma(-d, q, n), r, q);
}

// Whether that holds, for n > 0 and |d| >= 1e-14: 2^-500 <= n < 2^960 and |d| <
// 2^500 from the upper halves (then neither quotient nor residual underflows and
// nothing overflows), and a lower half of d that is not all ones.
OFB_HOST_DEVICE bool quotient_in_range(int n_hi, int d_hi, int d_lo) {
  constexpr unsigned kLow = (1023u - 500u) << 20, kHigh = (1023u + 960u) << 20, kMost = (1023u + 500u) << 20;
  return static_cast<unsigned>(n_hi) - kLow < kHigh - kLow && (static_cast<unsigned>(d_hi) & 0x7fffffffu) < kMost &&
         d_lo != -1;
}

}  // namespace ofb
