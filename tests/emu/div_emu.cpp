// Test-only CPU build of the shared division (cfdv_b200/csrc/divisor.h).  Used only by
// tests/test_divisor.py.
#include "../../cfdv_b200/csrc/divisor.h"

// q[i] = x[i] / d[i] through a Divisor of d[i]
extern "C" void emu_divide(const double* x, const double* d, double* q, long n) {
  for (long i = 0; i < n; i++) q[i] = cfdv::Divisor(d[i])(x[i]);
}
