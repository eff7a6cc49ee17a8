// fv3g_fp64.cuh -- FP64 values handled through their bit patterns.  FP64
// instructions run at 1/64 of the FP32 rate here (16 cycles of an SM per warp and
// instruction), and |a|, -a, min, max and comparisons of doubles are FP64
// instructions; the same on the high and low words runs in the integer pipe.
// Values are taken to be numbers: a NaN compares by its bits.  Where one may come in, a
// test on the high word goes beside the form, or chooses the FP64 one.
#pragma once

#include <cuda_runtime.h>

namespace fv3g {

__device__ __forceinline__ unsigned long long dbits(double a) { return (unsigned long long)__double_as_longlong(a); }
__device__ __forceinline__ double absv(double a) {
  return __hiloint2double(__double2hiint(a) & 0x7fffffff, __double2loint(a));
}
__device__ __forceinline__ double negv(double a) {
  return __hiloint2double(__double2hiint(a) ^ 0x80000000, __double2loint(a));
}
__device__ __forceinline__ double signed_as(double a, double b) {  // a >= 0 with the sign of b
  return __hiloint2double(__double2hiint(a) | (__double2hiint(b) & 0x80000000), __double2loint(a));
}
// a NaN as arithmetic leaves it (quiet); a value without a finite one
__device__ __forceinline__ bool is_nan(double a) { return 2u * (unsigned)__double2hiint(a) > 0xffe00000u; }
__device__ __forceinline__ bool inf_or_nan(double a) { return (__double2hiint(a) & 0x7ff00000) == 0x7ff00000; }
// of non-negative values
__device__ __forceinline__ bool mag_less(double a, double b) { return dbits(a) < dbits(b); }
__device__ __forceinline__ double mag_min(double a, double b) { return mag_less(a, b) ? a : b; }
__device__ __forceinline__ double mag_max(double a, double b) { return mag_less(a, b) ? b : a; }
// a 2^K for K = -2, -1, 1; zero, infinities, NaN and magnitudes below 2^-1019 as they are
template <int K>
__device__ __forceinline__ double scale2(double a) {
  const int hi = __double2hiint(a);
  const bool ok = 2u * (unsigned)hi - 0x00800000u < 0xff600000u;  // exponent field 4 .. 2046
  return __hiloint2double(ok ? hi + K * 0x00100000 : hi, __double2loint(a));
}
// |a| / 4; zero below 2^-1019, an infinity as it is, a NaN as it is with keep and zero without
__device__ __forceinline__ double quarter_mag(double a, bool keep) {
  const int hi = __double2hiint(a), mag = hi & 0x7fffffff;
  const unsigned t = 2u * (unsigned)hi - 0x00800000u;
  const bool ok = t <= 0xff600000u || keep;
  return __hiloint2double(ok ? (t < 0xff600000u ? mag - 0x00200000 : mag) : 0, ok ? __double2loint(a) : 0);
}
// 1 / x to within an ulp in three FP64 instructions (an IEEE division takes about
// eleven): an FP32 reciprocal r of the significand, then r + r (e + e^2) with e = 1 -
// x r, Householder's third-order step for 1/x (error e^3 ~ 2^-66).  Magnitudes
// outside 2^-999 .. 2^1001, zero, infinities and NaN divide.
__device__ __forceinline__ double fast_rcp(double x) {
  const int hi = __double2hiint(x), lo = __double2loint(x);
  const int ex = (hi >> 20) & 0x7ff;
  if ((unsigned)(ex - 24) > 2000u) return 1.0 / x;
  const double m = __hiloint2double((hi & 0x000fffff) | 0x3ff00000, lo);  // in [1, 2)
  const float rf = __fdividef(1.f, __int_as_float(0x3f800000 | (hi & 0x000fffff) << 3 | (unsigned)lo >> 29));
  const int fb = __float_as_int(rf);
  const double r0 = __hiloint2double((((fb >> 23) + 896) << 20) | (fb & 0x007fffff) >> 3, fb << 29);
  const double e = fma(negv(m), r0, 1.0);
  const double r = fma(fma(e, e, e), r0, r0);
  return __hiloint2double((__double2hiint(r) + ((1023 - ex) << 20)) ^ (hi & 0x80000000), __double2loint(r));
}
// a / b from the reciprocal with one residual correction (rounded correctly but for rare ties)
__device__ __forceinline__ double fast_div(double a, double b) {
  const int ex = (__double2hiint(b) >> 20) & 0x7ff;
  if ((unsigned)(ex - 24) > 2000u) return a / b;
  const double r = fast_rcp(b), q = a * r;
  return inf_or_nan(q) ? q : fma(fma(negv(q), b, a), r, q);  // (an infinite q has no residual)
}
// a != 0 by words (a test of the whole shifted pattern is compiled to an FP64 comparison)
__device__ __forceinline__ bool nonzero(double a) {
  return ((__double2hiint(a) & 0x7fffffff) | __double2loint(a)) != 0;
}
// a > 0, a < 0, a and b of opposite strict signs
__device__ __forceinline__ bool pos(double a) { return __double_as_longlong(a) > 0; }
__device__ __forceinline__ bool neg(double a) { return __double2hiint(a) < 0 && nonzero(a); }
__device__ __forceinline__ bool opp(double a, double b) {
  return (__double2hiint(a) ^ __double2hiint(b)) < 0 && nonzero(a) && nonzero(b);
}
// a < b (-0 below +0)
__device__ __forceinline__ long long dkey(double a) {
  const long long k = __double_as_longlong(a);
  return k ^ ((k >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ bool less(double a, double b) { return dkey(a) < dkey(b); }
// a into the range of x0 and x1, as fmin(fmax(a, lo), hi) has it: where a is NaN (as it is to be
// where x0 or x1 is) the lower one, or the number of the two
__device__ __forceinline__ double clamp_between(double a, double x0, double x1) {
  const bool up = less(x0, x1);
  const double lo = up ? x0 : x1, hi = up ? x1 : x0;
  const double in = less(a, lo) ? lo : less(hi, a) ? hi : a;
  return is_nan(a) ? (is_nan(lo) ? hi : lo) : in;
}
// a into the range of 0, x and y
__device__ __forceinline__ double clamp0(double a, double x, double y) {
  const double lx = __double2hiint(x) < 0 ? x : 0.0, hx = __double2hiint(x) < 0 ? 0.0 : x;
  const double lo = less(y, lx) ? y : lx, hi = less(hx, y) ? y : hx;
  return less(a, lo) ? lo : less(hi, a) ? hi : a;
}

}  // namespace fv3g
