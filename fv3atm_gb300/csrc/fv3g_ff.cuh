// fv3g_ff.cuh -- float-float arithmetic shared by the FP32 remap and the
// FP32 global mass sums.
#pragma once

#include <cuda_runtime.h>

#include "fv3g_pair.cuh"

namespace fv3g {

// Float-float arithmetic (an unevaluated sum of two floats, ~48-bit
// significand): the error-free transformations TwoSum (Knuth) and TwoProd
// (with fma), then one renormalisation.
struct FF {
  float hi, lo;
};
__device__ __forceinline__ FF ff_add(FF a, FF b) {
  const float s = a.hi + b.hi;
  const float bb = s - a.hi;
  float e = (a.hi - (s - bb)) + (b.hi - bb);
  e += a.lo + b.lo;
  const float h = s + e;
  return FF{h, e - (h - s)};
}
__device__ __forceinline__ FF ff_neg(FF a) { return FF{-a.hi, -a.lo}; }
__device__ __forceinline__ FF ff_prod(float a, float b) {
  const float p = a * b;
  return FF{p, fmaf(a, b, -p)};
}

// Two float-floats in lockstep (packed f32x2 instructions), each with the roundings
// of the forms above.
struct FFP {
  F2 hi, lo;
};
__device__ __forceinline__ FFP ffp_renorm(F2 s, F2 e) {
  const F2 h = add2(s, e);
  return FFP{h, sub2(e, sub2(h, s))};
}
__device__ __forceinline__ FFP ffp_add(FFP a, FFP b) {
  const F2 s = add2(a.hi, b.hi), bb = sub2(s, a.hi);
  return ffp_renorm(s, add2(add2(sub2(a.hi, sub2(s, bb)), sub2(b.hi, bb)), add2(a.lo, b.lo)));
}
__device__ __forceinline__ FFP ffp_sub(FFP a, FFP b) {
  const F2 s = sub2(a.hi, b.hi), bb = sub2(s, a.hi);
  return ffp_renorm(s, add2(sub2(sub2(a.hi, sub2(s, bb)), add2(b.hi, bb)), sub2(a.lo, b.lo)));
}
__device__ __forceinline__ FFP ffp_addf(FFP a, F2 b) {
  const F2 s = add2(a.hi, b), bb = sub2(s, a.hi);
  return ffp_renorm(s, add2(add2(sub2(a.hi, sub2(s, bb)), sub2(b, bb)), a.lo));
}
// (scalar: a packed product that feeds a packed addition is contracted into a packed
// multiply-add, which would count the product's low part twice)
__device__ __forceinline__ FFP ffp_prod(F2 a, float b) {
  const F2 p{__fmul_rn(a.x, b), __fmul_rn(a.y, b)};
  return FFP{p, F2{fmaf(a.x, b, -p.x), fmaf(a.y, b, -p.y)}};
}

// the exact product a * b * c of three floats as float-float (to ~2^-48):
// TwoProd of a*b, then of its leading part with c, the low part's product
// folded in with one fma
__device__ __forceinline__ FF ff_prod3(float a, float b, float c) {
  const FF ab = ff_prod(a, b);
  const float p = ab.hi * c;
  return FF{p, fmaf(ab.lo, c, fmaf(ab.hi, c, -p))};
}

}  // namespace fv3g
