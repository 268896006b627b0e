// xg_rcp.h -- the reciprocal on the pivot chains of the LDL' kernels.
#pragma once

#include <cuda_runtime.h>

namespace xg {

// 1/d with a short dependency chain: d's leading 24 bits re-encoded as a
// single-precision number by integer arithmetic (the exponent rebiased from
// 1023 to 127, no conversion instruction), the single-precision hardware
// reciprocal of that, re-encoded as a double, then one step of the
// cubically convergent reciprocal iteration in FP64,
// x1 = x0 (1 + e + e^2) with e = 1 - d x0 (the order-3 member of
// Householder's family for f(x) = 1/x - d: A. S. Householder, The Numerical
// Treatment of a Single Nonlinear Equation, McGraw-Hill 1970; the
// truncated series of 1/(1 - e)).  The relative error of x1 is e^3 plus
// the rounding of the two FMAs, so the seed's ~22 correct bits become more
// than double precision.  Outside 2^-100 .. 2^100 in magnitude the
// correctly rounded reciprocal is used.  The stored reciprocal pivots of
// the factorisations are the correctly rounded ones; this one only scales
// the columns during elimination.  xg_chain_reciprocal_check evaluates it
// beside __drcp_rn for the error-bound test.
#ifdef __CUDACC__
__device__ __forceinline__ double chain_reciprocal(double d) {
  const int hi = __double2hiint(d), lo = __double2loint(d);
  const int ahi = hi & 0x7fffffff;
  if (ahi < ((1023 - 100) << 20) || ahi >= ((1023 + 100) << 20)) return __drcp_rn(d);
  const unsigned fb = ((unsigned)hi & 0x80000000u) |
                      ((unsigned)(ahi - (896 << 20)) << 3) | ((unsigned)lo >> 29);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fb)));
  const unsigned rb = __float_as_uint(r);
  const int rhi = (int)((rb & 0x80000000u) | (((rb & 0x7fffffffu) >> 3) + (896u << 20)));
  const int rlo = (int)(rb << 29);
  const double x = __hiloint2double(rhi, rlo);
  const double e = fma(-d, x, 1.0);
  return fma(x, fma(e, e, e), x);
}
#endif

// 1/d in integer arithmetic, off the FP64 unit, for the tile LDL's chain of
// pivots: the single-precision hardware reciprocal y0 of d's leading 24 bits
// as a 24-bit integer, the exact residual e = 1 - m y0 of the 53-bit
// significand m in [1, 2) as a 64-bit integer (|e| < 2^-21, so the low 64 bits
// of the product hold it), then the same cubic step y1 = y0 (1 + e + e^2) in
// fixed point with 63 fraction bits, rounded to nearest.  Every discarded part
// lies below 2^-59 of the result, so it is within 0.505 ulp of 1/d.
// chain_reciprocal's three dependent FP64 operations on a unit that takes one
// per 64 cycles from a warp make 284 cycles; this takes 153.  It holds wherever
// d and 1/d are normal numbers (reciprocal_out_of_range tells where not); the
// caller looks where a branch costs it nothing.  The hardware's error of one
// unit may take the seed of a significand next to 2 below 1/2 (and next to 1
// to 1): it is held in [1/2, 1], where its 24 bits have one meaning.
// xg_pivot_reciprocal_check evaluates it on the device.
__device__ __forceinline__ bool reciprocal_out_of_range(double d) {
  const int be = (__double2hiint(d) >> 20) & 0x7ff;
  return be < 1 || be > 2044;
}
// from the bits rb of the seed
__device__ __forceinline__ double wide_reciprocal_from(double d, unsigned rb) {
  const int hi = __double2hiint(d);
  const unsigned lo = (unsigned)__double2loint(d);
  const int be = (hi >> 20) & 0x7ff;
  const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;   // m = (mh 2^32 + lo) 2^-52
  // y0 2^-24, in [1/2, 1]
  const unsigned y0 = rb >= 0x3f800000u ? 0x1000000u
                      : rb < 0x3f000000u ? 0x800000u : (rb & 0x7fffffu) | 0x800000u;
  const unsigned long long p = (unsigned long long)lo * y0;
  const unsigned ph = (unsigned)(p >> 32) + mh * y0;
  const long long e = -(long long)(((unsigned long long)ph << 32) | (unsigned)p);   // e 2^76
  const int eh = (int)(e >> 32);
  const long long c = (e + (((long long)eh * eh) >> 12) + 0x8000) >> 16;    // (e + e^2) 2^60
  const long long q = (long long)((unsigned long long)(unsigned)c * y0) +
                      (((long long)(int)(c >> 32) * (int)y0) << 32);
  const unsigned long long y = ((unsigned long long)y0 << 39) + (unsigned long long)(q >> 21);
  // y in (2^62, 2^63]: the leading bit adds itself to the exponent field
  return __longlong_as_double(
      (long long)((((unsigned long long)(2044 - be) << 52) + ((y + 512) >> 10)) |
                  ((unsigned long long)((unsigned)hi & 0x80000000u) << 32)));
}
#ifdef __CUDACC__
__device__ __forceinline__ double wide_reciprocal(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r)
      : "f"(__uint_as_float(0x3f800000u | ((hi & 0xfffffu) << 3) | (lo >> 29))));
  return wide_reciprocal_from(d, __float_as_uint(r));
}
#endif
}  // namespace xg
