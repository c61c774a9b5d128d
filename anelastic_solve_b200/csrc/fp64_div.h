// fp64_div.h -- quotients and reciprocals without a division in the chain.
// Plain C++ where nvcc does not compile it (the tests do that).
#pragma once

#include <cmath>
#include <cstring>

#ifdef __CUDACC__
#define ANEL_HD __host__ __device__ __forceinline__
#else
#define ANEL_HD inline
#endif

namespace anel {

// biased exponent
ANEL_HD unsigned fp64_exponent(double x) {
#ifdef __CUDA_ARCH__
  return (unsigned)(__double2hiint(x) >> 20) & 0x7ffu;
#else
  unsigned long long u;
  std::memcpy(&u, &x, sizeof(u));
  return (unsigned)(u >> 52) & 0x7ffu;
#endif
}

// The y that div_by takes with b: 1 / b, or NaN where |b| is not within
// 2^-100..2^100.
ANEL_HD double div_reciprocal(double b) { return fp64_exponent(b) - 923u <= 200u ? 1.0 / b : NAN; }

// a / b, correctly rounded, from y = 1 / b rounded to nearest: two
// corrections q <- q + (a - b q) y.  The first makes q faithful, and then the
// second gives the rounded quotient (Markstein, IBM J. Res. Dev. 34, 1990);
// outside the exponents where no step can over- or underflow, and for zero,
// infinite and NaN quotients, the division itself.
ANEL_HD double div_by(double a, double b, double y) {
  const double q0 = a * y;
  const double q1 = fma(fma(-b, q0, a), y, q0);
  const double q2 = fma(fma(-b, q1, a), y, q1);
  return fp64_exponent(q0) - 200u < 1600u ? q2 : a / b;
}

// 1 / x within a unit in the last place from an approximation y that is off
// by 2^-17 of it at most: two Newton steps y <- y + y (1 - x y), each
// squaring the error.
ANEL_HD double rcp_newton(double x, double y) {
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

}  // namespace anel
