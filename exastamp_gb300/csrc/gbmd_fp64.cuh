// gbmd_fp64.cuh -- square root, reciprocal and table knot of the plain-FP64 pair
// kernels, in few FP64 instructions (each takes 16 cycles of an SM a warp; the
// library's square root and division take some 20 to 30).
#pragma once
#include "gbmd_internal.cuh"

namespace gbmd {

// r = sqrt(d2), and 1/r with it where INV.  The FP32 rsqrt is the seed y0; with
// e = 1 - d2 y0^2, below 2^-20, one step of Householder's method of third order for
// 1/y^2 = d2 (the binomial series of (1 - e)^(-1/2) up to e^2) gives
//   y = y0 (1 + e/2 + 3 e^2/8),   remainder 5 e^3/16, below 2^-61,
// Newton's method for r^2 = d2 (Heron's), its division replaced by y/2, corrects
// r = d2 y, and Newton's for 1/y = r corrects y.  Both corrections form their
// residual with one rounding (fma), so r and y end within one unit in the last
// place: half from the last rounding, the rest below 2^-20 of one.  Outside the
// range that FP32 covers the library functions are taken.
// (A. S. Householder, The Numerical Treatment of a Single Nonlinear Equation, 1970.)
template <bool INV>
__device__ __forceinline__ double root(double d2, double& y) {
  const uint32_t hi = (uint32_t)__double2hiint(d2);
  if (hi - 0x3a000000u < 0x0c000000u) {  // 2^-95 <= d2 < 2^97
    const float s = __uint_as_float(((hi - 0x38000000u) << 3) | ((uint32_t)__double2loint(d2) >> 29));
    const double y0 = widen(rsqrtf(s));
    const double e = fma(-(d2 * y0), y0, 1.0);
    y = fma(y0 * e, fma(e, 0.375, 0.5), y0);
    double r = d2 * y;
    r = fma(fma(-r, r, d2), 0.5 * y, r);
    if (INV) y = fma(fma(-r, y, 1.0), y, y);
    return r;
  }
  const double r = sqrt(d2);
  y = 1.0 / r;
  return r;
}

// 1/d2: the FP32 reciprocal as seed y0 and one step of Householder's method of
// third order for 1/y = d2, which for the reciprocal is the geometric series of
// 1/(1 - e), e = 1 - d2 y0, up to e^2: y0 (1 + e + e^2), remainder e^3.  e is below
// 2^-22, so the remainder is below 2^-66 and the last rounding is all that counts:
// within one unit in the last place.
__device__ __forceinline__ double inverse(double d2) {
  const uint32_t hi = (uint32_t)__double2hiint(d2);
  if (hi - 0x3a000000u < 0x0c000000u) {
    const float s = __uint_as_float(((hi - 0x38000000u) << 3) | ((uint32_t)__double2loint(d2) >> 29));
    const double y0 = widen(__frcp_rn(s));
    const double e = fma(-d2, y0, 1.0);
    return fma(y0, fma(e, e, e), y0);
  }
  return 1.0 / d2;
}

// Knot m = floor(t), capped at nr - 1, and p = t - m, capped at 1: the integer
// part of t in [1, 2^20) by shifts, the fraction by one subtraction.
__device__ __forceinline__ int r_knot_d(double t, int nr, double& p) {
  const long long b = __double_as_longlong(t);
  const int ex = (int)(b >> 52) - 1023;
  if ((unsigned)ex < 20u) {
    const long long mant = b & 0xfffffffffffffll;
    const int m = (int)((mant | 0x10000000000000ll) >> (52 - ex));
    if (m < nr) {
      p = __longlong_as_double(((mant << ex) & 0xfffffffffffffll) | 0x3ff0000000000000ll) - 1.0;
      return m;
    }
  }
  const int m = min((int)t, nr - 1);
  p = fmin(t - m, 1.0);
  return m;
}

}  // namespace gbmd
