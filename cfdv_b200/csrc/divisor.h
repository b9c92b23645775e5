// Division by a value that many quotients share, for the device and, in tests, the host.
#pragma once

#include <cmath>
#include <cstring>

#ifdef __CUDACC__
#define CFDV_DIV_HD __host__ __device__ __forceinline__
#else
#define CFDV_DIV_HD inline
#endif

namespace cfdv {

// x / d with the reciprocal of d at hand: one Newton correction of the quotient (Markstein's
// final step) gives the correctly rounded quotient but for rare last-bit cases, in 3 operations;
// the compiled division takes about 35 instructions, 3 to 8 us a pass B of 1.38M unknowns.
// Numerators and reciprocals between 2^-465 and 2^465 (about 1e-140 and 1e140) only: no product
// below leaves the normal numbers then, the residual of about 2^-53 x among them.  A zero's quotient is
// the first product, its sign with it (Dirichlet rows are zeros: sent to the division they cost a mixed
// solve 1%); anything else (infinite, NaN, tiny, huge) takes the division itself.  A numerator's range
// is read off its exponent's word: two comparisons of the value cost FP64 solves of 16,800 to 72,000
// hexes 0.4 to 0.9%.
struct Divisor {
  double d, rd;
  bool fast;
  CFDV_DIV_HD explicit Divisor(double v) : d(v), rd(1.0 / v), fast(fabs(rd) >= 1e-140 && fabs(rd) <= 1e140) {}
  CFDV_DIV_HD static bool ordinary(double v) {
    unsigned long long b;
    memcpy(&b, &v, sizeof(b));
    return ((unsigned)(b >> 32) & 0x7fffffffu) - ((1023u - 465u) << 20) < (930u << 20);
  }
  CFDV_DIV_HD double operator()(double x) const {
    const double q = x * rd;
    if (!(fast && (ordinary(x) || x == 0.0))) return x / d;
    return x == 0.0 ? q : fma(fma(-q, d, x), rd, q);
  }
};

}  // namespace cfdv
