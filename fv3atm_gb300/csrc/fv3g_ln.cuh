// fv3g_ln.cuh -- ln p of pressures by table, for the interface pressures of the field
// remaps in ln p (fv3g_remap.cu).
#pragma once

#include <cuda_runtime.h>

namespace fv3g {

constexpr int LN_N = 1024;  // table entries: one per 2^-10 of the significand

// ln p by table (Tang 1990): the significand m in [0.75, 1.5) times the tabulated
// reciprocal r of its bin leaves 1 + e with |e| < 2^-10, and ln p = k ln 2 - ln r + ln(1 +
// e), the last as its Taylor polynomial of degree 6 (error 2^-63 relative).  k ln 2 is split so
// that its leading part is exact.  From p = 3 on and below 3/16 the result is above 1 in magnitude,
// and the errors of the tabulated term (an ulp of a value below 0.41 at most), of the inner sum
// and of the last rounding stay below 0.9 of its ulp (0.56 from 1 to 110 kPa, measured); between, where
// the term is as large as the result (1.5 ulp beside 1), and for zero, negative, subnormal, infinite
// and NaN p, log runs: a level or two of a column.
__device__ __forceinline__ double ln_tab(double p, const double2* tab) {
  const int hi = __double2hiint(p);
  if ((unsigned)(hi - 0x00100000) >= 0x7fe00000u || (unsigned)(hi - 0x3fc80000) < 0x00400000u) return log(p);
  const int up = (hi >> 19) & 1;  // significand from 1.5 on: halved
  const float kf = (float)((hi >> 20) - 1023 + up);
  const unsigned kb = __float_as_uint(kf);
  const double k = __hiloint2double(kf == 0.f ? 0 : (int)(((kb & 0x7fffffffu) >> 3) + (896u << 20) | (kb & 0x80000000u)),
                                    (int)(kb << 29));
  const double m = __hiloint2double((hi & 0x000fffff) | (up ? 0x3fe00000 : 0x3ff00000), __double2loint(p));
  const double2 t = tab[(hi >> 10) & (LN_N - 1)];
  const double e = fma(m, t.x, -1.0);
  double c = fma(e, -1.0 / 6.0, 1.0 / 5.0);
  c = fma(e, c, -1.0 / 4.0);
  c = fma(e, c, 1.0 / 3.0);
  c = fma(e, c, -0.5);
  const double l = fma(e * e, c, e);
  constexpr double LN2_HI = 0x1.62e42fefa38p-1, LN2_LO = 0x1.ef35793c7673p-45;  // ln 2: 42 bits and the rest
  return fma(k, LN2_HI, t.y + fma(k, LN2_LO, l));
}
__device__ __forceinline__ void ln_table(double2* tab) {
  for (int i = threadIdx.x; i < LN_N; i += blockDim.x) {
    const float c = 1.f + (i + 0.5f) / LN_N;  // the bin's middle; halved from 1.5 on
    const double r = (double)(1.f / (i >= LN_N / 2 ? 0.5f * c : c));
    tab[i] = make_double2(r, -log(r));
  }
  __syncthreads();
}

}  // namespace fv3g
