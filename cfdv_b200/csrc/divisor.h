// Division by a value that many quotients share, for the device and, in tests, the host.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define CFDV_DIV_HD __host__ __device__ __forceinline__
#else
#define CFDV_DIV_HD inline
#endif

namespace cfdv {

// x / d with the reciprocal of d at hand: one Newton correction of the quotient (Markstein's
// final step) gives the correctly rounded quotient but for rare last-bit cases, in 3 operations;
// the compiled division takes about 35 instructions, 3 to 8 us a pass B of 1.38M unknowns.
// Numerators and reciprocals of ordinary size only: no product below leaves the normal numbers then,
// the residual of about 2^-53 x among them.  A zero's quotient is the first product, its sign with it;
// for anything else (infinite, NaN, tiny, huge) the division itself.
struct Divisor {
  static constexpr double kLow = 1e-140, kHigh = 1e140;
  double d, rd;
  bool fast;
  CFDV_DIV_HD explicit Divisor(double v) : d(v), rd(1.0 / v), fast(fabs(rd) >= kLow && fabs(rd) <= kHigh) {}
  CFDV_DIV_HD double operator()(double x) const {
    const double ax = fabs(x), q = x * rd;
    if (!(fast && ((ax >= kLow && ax <= kHigh) || ax == 0.0))) return x / d;
    return ax == 0.0 ? q : fma(fma(-q, d, x), rd, q);
  }
};

}  // namespace cfdv
