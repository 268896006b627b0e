// Host driver for tests/test_pivot_reciprocal.py: xg::wide_reciprocal_from on the
// host, with a given seed.
#include <cuda_runtime.h>

#include <cstring>

namespace {
unsigned long long bits(double v) {
  unsigned long long u;
  std::memcpy(&u, &v, 8);
  return u;
}
int __double2hiint(double v) { return (int)(bits(v) >> 32); }
int __double2loint(double v) { return (int)(bits(v) & 0xffffffffu); }
double __longlong_as_double(long long u) {
  double v;
  std::memcpy(&v, &u, 8);
  return v;
}
}  // namespace

#include "../../xara_gb300/csrc/xg_rcp.h"

extern "C" void reciprocals(int n, const double *d, const unsigned *seed, double *y) {
  for (int i = 0; i < n; i++) y[i] = xg::wide_reciprocal_from(d[i], seed[i]);
}
