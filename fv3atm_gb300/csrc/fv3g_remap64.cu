// fv3g_remap64.cu -- Lagrangian-to-Eulerian column remap of FP64 fields, one
// warp per column (map_scalar / map1_ppm with cs_profile and ppm_profile of
// fv_mapz.F90, GFDL_atmos_cubed_sphere, absent submodule .gitmodules:1-4).
//
// The schemes and the division of a column among lanes are those of
// k_remap_warp (fv3g_remap.cu), which keeps FP32.  Here the FP64 pipe is the
// bound (1/64 of the FP32 rate), so the kernel counts FP64 instructions per
// layer and field:
//   * whatever depends on the column alone is formed once for all its fields:
//     the interface system's rows scaled by their pivots (three multiply-adds per
//     interface and field, two for back substitution and scans), kord 4's slopes
//     and interfaces as linear forms (it divided about twelve times per layer and
//     field), and every target layer's mean as w1 (v + S1 h + Q1 s) + w2 (v' + S2 h'
//     + Q2 s') over the two source layers at its ends (target thickness, squares
//     and sums of the overlap fractions folded into the weights);
//   * min, max, signs, comparisons and halvings run on bit patterns in the
//     integer pipe;
//   * the positivity test compares |bl + br| with the mean's height above the
//     floor first: the parabola's minimum lies no lower than q - |bl + br|.
// These forms take ordinary numbers; a column that holds others goes through the schemes
// in their FP64 forms (general_fields), found by an integer test per value and one vote per
// field.
// A call's divisions (pressures, pivots, target thicknesses) take fast_rcp and
// fast_div (fv3g_fp64.cuh), a third and a half of the FP64 instructions of an IEEE
// division.  Measured: the remap of 6 x C96 L64 x 4 tracers, kord 4, 13.2 -> 2.9 ms
// (with 4 layers a lane for any level count and IEEE divisions 5.6); of 6 x C192 L127 x
// 9, kord 9, 35 ms (a step 238 -> 172 with it).  Five layers a lane (128 levels and more)
// spill 76 bytes at kord 9 at the 168 registers that three CTAs leave.
#include <algorithm>
#include <mutex>

#include "fv3g_fp64.cuh"
#include "fv3g_internal.cuh"
#include "fv3g_profile.cuh"
#include "fv3g_remap.cuh"

namespace fv3g {
namespace {

constexpr int COLS = 4;   // columns (warps) per CTA: 4 FP64 columns are one 32-byte sector
constexpr int SLOTS = 3;  // fields in the shared-memory ring
constexpr int MAX_FIELDS = 32 * 32;  // fields of a launch: a bit of a lane's word each (general_fields)
constexpr unsigned FULL = 0xffffffffu;

// one pad element per 16 levels: blocked lane ownership hits distinct banks
__host__ __device__ constexpr int pd(int k) { return k + (k >> 4); }

template <int NPL>
struct Col64 {
  static constexpr int N = pd(32 * NPL) + 1;
  double pe1[N], dp[N];
  double l[N], h[N], s[N];            // parabola of every source layer: left edge, (r - l + s6) / 2, -s6 / 3
  double w1[N], S1[N], Q1[N];         // weights of every target layer's mean
  double w2[N], S2[N], Q2[N];
};
template <int NPL>
__host__ __device__ constexpr int ring_pitch64() {
  int p = pd(32 * NPL) + 1;
  while (p % 16 != 4) ++p;  // the 4 columns of one copy instruction on distinct banks
  return p;
}
template <int NPL>
constexpr size_t smem64() {
  return COLS * sizeof(Col64<NPL>) + (size_t)SLOTS * COLS * ring_pitch64<NPL>() * sizeof(double);
}

template <int W>
__device__ __forceinline__ void pending() { asm volatile("cp.async.wait_group %0;\n" ::"n"(W) : "memory"); }

// m2 * m1 (m1 applied first) of 2x2 matrices, rescaled by a power of two
struct M2 {
  double a, b, c, d;
};
__device__ __forceinline__ M2 after(const M2& m2, const M2& m1) {
  M2 r{fma(m2.a, m1.a, m2.b * m1.c), fma(m2.a, m1.b, m2.b * m1.d), fma(m2.c, m1.a, m2.d * m1.c),
       fma(m2.c, m1.b, m2.d * m1.d)};
  const double m = mag_max(mag_max(absv(r.a), absv(r.b)), mag_max(absv(r.c), absv(r.d)));
  const long long e = (__double_as_longlong(m) >> 52) & 0x7ff;
  const double s = __longlong_as_double((2046 - e) << 52);
  r.a *= s; r.b *= s; r.c *= s; r.d *= s;
  return r;
}
__device__ __forceinline__ M2 up(const M2& m, int o) {
  return M2{__shfl_up_sync(FULL, m.a, o), __shfl_up_sync(FULL, m.b, o), __shfl_up_sync(FULL, m.c, o),
            __shfl_up_sync(FULL, m.d, o)};
}

// kord 9: the limited value of raw interface a between layers of means qa and
// qb; dl, dc, dr: the jumps across the interfaces before, at and after it
__device__ __forceinline__ double limit9(double a, double qa, double qb, double dl, double dr, int iv, double floor_v) {
  const bool up_ = less(qa, qb);
  const double lo = up_ ? qa : qb, hi = up_ ? qb : qa;
  const bool mono = (pos(dl) && pos(dr)) || (neg(dl) && neg(dr));
  const double lower = less(a, lo) ? lo : a, upper = less(hi, a) ? hi : a;
  const double below = iv >= 0 && less(upper, floor_v) ? floor_v : upper;
  return mono ? (less(hi, lower) ? hi : lower) : (pos(dl) ? lower : below);
}

// Whether a's magnitude is ordinary: 2^-999 .. 2^977 (so neither zero, infinite nor NaN).
__device__ __forceinline__ bool ordinary(double a) {
  return (unsigned)(((__double2hiint(a) >> 20) & 0x7ff) - 24) <= 1976u;
}
__device__ __forceinline__ bool huge_or_nan(double a) { return (__double2hiint(a) & 0x7ff00000) >= 0x7d000000; }

// The fields (bit f / 32 of lane f % 32's word) whose columns hold something else than
// ordinary numbers -- a layer or target without thickness, infinities, NaN -- once more by
// the schemes in their FP64 forms (fv3g_profile.cuh), whose minima and maxima take the number
// beside a NaN; the overlaps come from the pressures one by one.  Rare, and called when no
// column constant is held any more, so that the field loop keeps its registers; in that
// loop the same as a branch spilled 36 to 400 bytes.  One warp.
template <int KORD, int NPL>
__device__ __noinline__ void general_fields(Col64<NPL>& S, double* Q, unsigned fields, long long qo, int col, int lane,
                                            bool real, const RemapArgs<double>& a) {
  const int km = a.km, kn = a.kn, u0 = lane * NPL, nc = (int)a.ncol;
  const double floor_v = a.iv == 1 ? a.q_min : 0.0, qsv = a.qs ? a.qs[col] : 0.0, ps = S.pe1[pd(km)];
  auto q = [Q, km](int k) -> double { return Q[pd(min(max(k, 0), km - 1))]; };
  auto h = [&S, km](int k) -> double { return S.dp[pd(min(max(k, 0), km - 1))]; };
  double *const cp = S.w1, *const rd = S.S1;  // kord 9: the interface system's elimination, row by row
  __syncwarp();
  double lo_b = 0.0, gb = 0.0;
  if (KORD == 9 && km > 1) {
    gb = h(km - 2) / h(km - 1);
    lo_b = a.iv == -2 ? 0.0 : gb + 1.0;
    if (lane == 0) {
      const double g = h(1) / h(0);
      double c = (g + 1.0) / g;
      cp[0] = c;
      rd[0] = 1.0 / g;
      for (int u = 1; u < km; ++u) {
        const double d = h(u - 1) / h(u), r = 1.0 / (2.0 * (1.0 + d) - c);
        c = d * r;
        cp[pd(u)] = c;
        rd[pd(u)] = r;
      }
      rd[pd(km)] = 1.0 / ((a.iv == -2 ? 1.0 : gb) - lo_b * c);
    }
  }
  for (int f = 0; f < a.nfield; ++f) {
    if (!(__shfl_sync(FULL, fields, f & 31) >> (f >> 5) & 1)) continue;
    const double* src = a.q_in + qo + f * a.sQq;
    for (int k = lane; k < km; k += 32) Q[pd(k)] = src[(long long)k * a.sQk];
    __syncwarp();
    if (KORD == 9 && km > 1 && lane == 0) {
      const double g = h(1) / h(0);
      double y = ((g * (2.0 * g + 3.0)) * q(0) + q(1)) / (g + 1.0) * rd[0];
      S.l[0] = y;
      for (int u = 1; u < km; ++u) {
        y = (3.0 * (q(u - 1) + h(u - 1) / h(u) * q(u)) - y) * rd[pd(u)];
        S.l[pd(u)] = y;
      }
      const double r = a.iv == -2 ? qsv : ((gb * (2.0 * gb + 3.0)) * q(km - 1) + q(km - 2)) / (gb + 1.0);
      y = (r - lo_b * y) * rd[pd(km)];
      S.l[pd(km)] = y;
      for (int u = km - 1; u >= 0; --u) S.l[pd(u)] = y = S.l[pd(u)] - cp[pd(u)] * y;
    }
    if (KORD == 4)
      for (int k = u0; k < min(u0 + NPL, km); ++k) S.s[pd(k)] = ppm_slope_f<double>(k, km, q, h);
    __syncwarp();
    for (int u = u0; u < min(u0 + NPL, km + 1); ++u) {
      double v;
      if (km == 1) v = q(0);
      else if (KORD == 9) v = k9_interface_f(S.l[pd(u)], u, km, a.iv, floor_v, q);
      else
        v = ppm_interface<double>(u, km, a.iv, qsv, u >= 1 ? S.s[pd(u - 1)] : 0.0, u < km ? S.s[pd(u)] : 0.0, q, h);
      S.h[pd(u)] = v;
    }
    __syncwarp();
    Profile<double> p[NPL];
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
      const int k = u0 + j;
      if (k < km)
        p[j] = layer_profile_f<double, KORD>(k, km, q(k), S.h[pd(k)], S.h[pd(k + 1)], KORD == 9 ? 0.0 : S.s[pd(k)],
                                             a.iv, floor_v, q);
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < NPL; ++j)
      if (u0 + j < km) {
        const int i = pd(u0 + j);
        S.l[i] = p[j].l;
        S.h[i] = p[j].r;
        S.s[i] = p[j].s6;
      }
    __syncwarp();
    auto pe2_at = [&](int k) -> double {
      return a.pe2 != nullptr ? a.pe2[(long long)k * nc + col] : a.ak[k] + a.bk[k] * ps;
    };
    auto locate = [&](int k2, int& L, double& X) {
      const double pt = pe2_at(k2);
      L = min(k2, km - 1);
      while (L > 0 && S.pe1[pd(L)] > pt) --L;
      while (L < km - 1 && S.pe1[pd(L + 1)] <= pt) ++L;
      X = (pt - S.pe1[pd(L)]) / (S.pe1[pd(L + 1)] - S.pe1[pd(L)]);
    };
    auto mean = [&](int L, double x1, double x2) { return pmean(S.l[pd(L)], S.h[pd(L)], S.s[pd(L)], x1, x2); };
    for (int t = u0; t < min(u0 + NPL, kn); ++t) {
      int Lt, Lb;
      double Xt, Xb, out;
      locate(t, Lt, Xt);
      locate(t + 1, Lb, Xb);
      if (Lb == Lt || (Lb == Lt + 1 && Xb == 0.0)) {
        out = Xt == 0.0 && (Lb == Lt + 1 || Xb == 1.0) ? q(Lt) : mean(Lt, Xt, Lb == Lt ? Xb : 1.0);
      } else {
        double mass = Xt == 0.0 ? q(Lt) * h(Lt) : (h(Lt) * (1.0 - Xt)) * mean(Lt, Xt, 1.0);
        for (int m = Lt + 1; m < Lb; ++m) mass = mass + q(m) * h(m);
        if (Xb >= 1.0) mass = mass + q(Lb) * (h(Lb) * Xb);
        else if (Xb > 0.0) mass = mass + (h(Lb) * Xb) * mean(Lb, 0.0, Xb);
        out = mass * (1.0 / (a.dp2 ? a.dp2[(long long)t * nc + col] : pe2_at(t + 1) - pe2_at(t)));
      }
      if (real) a.q_out[qo + f * a.sQqo + (long long)t * a.sQk] = out;
    }
    __syncwarp();
  }
}

template <int KORD, int NPL>
__global__ void __launch_bounds__(32 * COLS, 3) k_remap64(const __grid_constant__ RemapArgs<double> a) {
  constexpr int RP = ring_pitch64<NPL>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Col64<NPL>& S = reinterpret_cast<Col64<NPL>*>(smem_raw)[warp];
  double* const ring = reinterpret_cast<double*>(smem_raw + COLS * sizeof(Col64<NPL>));
  const int nc = (int)a.ncol;
  const int col0 = blockIdx.x * COLS;
  const bool real = col0 + warp < nc;  // the last CTA's surplus warps repeat the last column and store nothing
  const int col = real ? col0 + warp : nc - 1;
  auto offsets = [&a](int c, long long& fo_, long long& qo_) {
    const unsigned ni = (unsigned)a.ni, nj = (unsigned)a.nj;
    const unsigned rest = (unsigned)c / ni, ci = (unsigned)c - rest * ni;
    const unsigned ct = rest / nj, cj = rest - ct * nj;
    fo_ = ct * a.sFt + a.pg.at(a.i1 + ci, a.j1 + cj);
    qo_ = ct * a.sQt + a.pg.at(a.i1 + ci, a.j1 + cj);
  };
  long long fo, qo;
  offsets(col, fo, qo);
  const int km = a.km, kn = a.kn, u0 = lane * NPL;

  // cooperative field copy: this thread's column and levels
  const int cc = threadIdx.x % COLS, kk = threadIdx.x / COLS;
  long long fo_c, qo_c;
  offsets(min(col0 + cc, nc - 1), fo_c, qo_c);
  auto issue = [&](int f) {
    if (f < a.nfield) {
      const double* src = a.q_in + qo_c + f * a.sQq;
      double* dst = ring + ((f % SLOTS) * COLS + cc) * RP;
#pragma unroll
      for (int r = 0; r < NPL; ++r) {
        const int k = kk + 32 * r;
        if (k < km) copy_async(dst + pd(k), src + (long long)k * a.sQk);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  issue(0);
  issue(1);

  // ------------------------------------------------ interface pressures pe1
  if (a.pe1 != nullptr) {
#pragma unroll
    for (int j = 0; j < NPL; ++j)
      if (u0 + j <= km) S.pe1[pd(u0 + j)] = a.pe1[(long long)(u0 + j) * nc + col];
  } else {
    const double ptop = a.ak[0];
    double dl[NPL], tot = 0.0;
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
      dl[j] = (u0 + j < km) ? a.dp[fo + (long long)(u0 + j) * a.sFk] : 0.0;
      tot += dl[j];
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double p = __shfl_up_sync(FULL, tot, o);
      if (lane >= o) tot = p + tot;
    }
    const double excl = __shfl_up_sync(FULL, tot, 1);  // sum over lower lanes
    double s = lane == 0 ? ptop : ptop + excl;
    if (lane == 0) S.pe1[0] = ptop;
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
      s += dl[j];
      if (u0 + j < km) S.pe1[pd(u0 + j + 1)] = s;
    }
  }
  __syncwarp();
  const double ps = S.pe1[pd(km)];
  auto pe2_at = [&](int k) -> double {
    if (a.pe2 != nullptr) return a.pe2[(long long)k * nc + col];
    return a.ak[k] + a.bk[k] * ps;
  };
#pragma unroll
  for (int j = 0; j < NPL; ++j)
    if (u0 + j < km) S.dp[pd(u0 + j)] = S.pe1[pd(u0 + j + 1)] - S.pe1[pd(u0 + j)];
  __syncwarp();

  // ------------------------------- overlap schedule and the targets' weights
  // Source layer holding target interface p (a short walk from the target's own
  // index) and p's fraction of it; Lt | Lb << 8 per target layer, bits 16 and 17:
  // the first / the last overlap is a whole layer.
  unsigned sched[NPL];
  unsigned general = 0;  // fields for general_fields
  bool odd = false;      // all of them
#pragma unroll
  for (int j = 0; j < NPL; ++j)
    if (u0 + j < km) odd |= !ordinary(S.dp[pd(u0 + j)]);
  {
    int L0 = 0;
    double X0 = 0.0, p0 = 0.0;
#pragma unroll
    for (int j = 0; j <= NPL; ++j) {
      const int k2 = min(u0 + j, kn);
      const double p = pe2_at(k2);
      int k1 = min(k2, km - 1);
      while (k1 > 0 && less(p, S.pe1[pd(k1)])) --k1;
      while (k1 < km - 1 && !less(p, S.pe1[pd(k1 + 1)])) ++k1;
      const double pl = S.pe1[pd(k1)], ph = S.pe1[pd(k1 + 1)];
      const double X = fast_div(p - pl, ph - pl);
      const int t = u0 + j - 1;
      if (j > 0) {
        unsigned sc = 0;
        if (t < kn) {
          const double dpk = a.dp2 ? a.dp2[(long long)t * nc + col] : p - p0;
          if (real && a.dp_out != nullptr) a.dp_out[fo + (long long)t * a.sFk] = dpk;
          odd |= !ordinary(dpk) | huge_or_nan(X0) | huge_or_nan(X);
          const bool inside = k1 == L0 || (k1 == L0 + 1 && !nonzero(X));
          const double x2 = inside && k1 == L0 ? X : 1.0;  // the first overlap's end
          const bool whole = !nonzero(X0) && (!inside || k1 == L0 + 1 || dbits(X) == dbits(1.0));
          const double rd = fast_rcp(dpk), dpt = S.dp[pd(L0)], dpb = S.dp[pd(k1)];
          const int i = pd(t);
          S.w1[i] = inside ? 1.0 : (dpt * (1.0 - X0)) * rd;
          S.S1[i] = whole ? 0.0 : X0 + x2;
          S.Q1[i] = whole ? 0.0 : fma(X0, X0 + x2, x2 * x2);
          const bool full = !inside && !less(X, 1.0);
          S.w2[i] = inside ? 0.0 : (dpb * X) * rd;
          S.S2[i] = full ? 0.0 : X;
          S.Q2[i] = full ? 0.0 : X * X;
          sc = (unsigned)L0 | (unsigned)(inside ? L0 : k1) << 8 | (whole ? 1u << 16 : 0u) | (full ? 1u << 17 : 0u);
          // whole layers between the two ends share one factor
          if (!inside && k1 > L0 + 1) sc |= 1u << 18;
        }
        sched[j - 1 >= 0 ? j - 1 : 0] = sc;
      }
      L0 = k1;
      X0 = X;
      p0 = p;
    }
  }
  auto rdpk_of = [&](int t) -> double {  // rare: layers spanning more than two source layers
    return 1.0 / (a.dp2 ? a.dp2[(long long)t * nc + col] : pe2_at(t + 1) - pe2_at(t));
  };

  const double floor_v = (a.iv == 1) ? a.q_min : 0.0;
  const double qsv = a.qs ? a.qs[col] : 0.0;
  odd = __any_sync(FULL, odd | huge_or_nan(qsv) | huge_or_nan(floor_v));
  // ------------------------------------------------ the column's linear forms
  // kord 9: y_u = e1 q_a + e2 q_b + aj y_{u-1} (layers a, b = u-1, u; top row 0, 1;
  // bottom row km-1, km-2), a_u = y_u - cp a_{u+1}; mf, mb: the multipliers of the
  // five steps of the forward and backward scans.
  // kord 4: slope of layer u: e1 D_{u+1} + e2 D_u before its limits; interface u:
  // q_{u-1} + aj D_u + cp dm_{u-1} - c2 dm_u inside, aj q_{u-1} + cp q_u + c2 q3 at u =
  // 1 and km-1 (q3: the layer beyond).
  double e1[NPL], e2[NPL], aj[NPL], cp[NPL], c2[NPL], mf[5], mb[5];
#pragma unroll
  for (int j = 0; j < NPL; ++j) e1[j] = e2[j] = aj[j] = cp[j] = c2[j] = 0.0;
  if (KORD == 9 && km > 1) {
    const double g = S.dp[pd(1)] / S.dp[0];
    double dd[NPL];
    M2 m{1.0, 0.0, 0.0, 1.0};
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
      const int u = u0 + j;
      dd[j] = (u >= 1 && u < km) ? fast_div(S.dp[pd(u - 1)], S.dp[pd(u)]) : 0.0;
      if (u >= 1 && u < km) m = after(M2{0.0, dd[j], -1.0, 2.0 * (1.0 + dd[j])}, m);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const M2 p = up(m, o);
      if (lane >= o) m = after(m, p);
    }
    const M2 e = up(m, 1);
    const double cp0 = (g + 1.0) / g;
    double cprev = (e.a * cp0 + e.b) / (e.c * cp0 + e.d);  // of interface u0-1 (lanes >= 1)
    const double gb = S.dp[pd(km - 2)] / S.dp[pd(km - 1)];
    const double lo_b = a.iv == -2 ? 0.0 : gb + 1.0;
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
      const int u = u0 + j;
      if (u == 0) {
        cp[j] = cp0;
        e1[j] = (g * (2.0 * g + 3.0)) / (g + 1.0) / g;
        e2[j] = 1.0 / (g + 1.0) / g;
      } else if (u < km) {
        const double rd = fast_rcp(2.0 * (1.0 + dd[j]) - cprev);
        cp[j] = dd[j] * rd;
        aj[j] = -rd;
        e1[j] = 3.0 * rd;
        e2[j] = 3.0 * dd[j] * rd;
      } else if (u == km) {
        const double rd = 1.0 / ((a.iv == -2 ? 1.0 : gb) - lo_b * cprev);
        aj[j] = -lo_b * rd;
        if (a.iv != -2) {
          e1[j] = (gb * (2.0 * gb + 3.0)) / (gb + 1.0) * rd;
          e2[j] = 1.0 / (gb + 1.0) * rd;
        }
      }
      cprev = cp[j];
    }
    double alf = 1.0, alb = 1.0;
#pragma unroll
    for (int j = 0; j < NPL; ++j) alf = aj[j] * alf;
#pragma unroll
    for (int j = NPL - 1; j >= 0; --j) alb = -cp[j] * alb;
#pragma unroll
    for (int o = 1, s = 0; o < 32; o <<= 1, ++s) {
      mf[s] = alf;
      mb[s] = alb;
      const double pa = __shfl_up_sync(FULL, alf, o), pb = __shfl_down_sync(FULL, alb, o);
      if (lane >= o) alf = alf * pa;
      if (lane + o < 32) alb = alb * pb;
    }
  }
  if (KORD == 4 && km > 1) {
    auto H = [&](int k) { return S.dp[pd(min(max(k, 0), km - 1))]; };
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
      const int u = u0 + j;
      const double hm = H(u - 2), h0 = H(u - 1), h1 = H(u), h2 = H(u + 1);
      const double pair = fast_rcp(h0 + h1);  // of interface u; the next one's is formed again
      if (u >= 1 && u <= km - 2) {            // CW84 eq. 1.7 slope
        const double f = h1 * fast_rcp(h0 + h1 + h2);
        e1[j] = f * ((2.0 * h0 + h1) * fast_rcp(h2 + h1));
        e2[j] = f * ((h1 + 2.0 * h2) * pair);
      }
      if (u >= 2 && u <= km - 2) {  // CW84 eq. 1.6 interface
        const double sall = fast_rcp(hm + h0 + h1 + h2);
        const double fa = (hm + h0) * fast_rcp(2.0 * h0 + h1), fb = (h2 + h1) * fast_rcp(2.0 * h1 + h0);
        aj[j] = h0 * pair + 2.0 * h1 * h0 * pair * (fa - fb) * sall;
        c2[j] = 2.0 * h0 * fa * sall;
        cp[j] = 2.0 * h1 * fb * sall;
      } else if (km == 2 && u == 1) {
        aj[j] = H(1) / (H(0) + H(1));
        cp[j] = H(0) / (H(0) + H(1));
      } else if (u == 1 || u == km - 1) {  // parabola through the three layers at the end
        const double h0 = u == 1 ? H(0) : H(km - 1), h1 = u == 1 ? H(1) : H(km - 2), h2 = u == 1 ? H(2) : H(km - 3);
        const double w0 = h1 * (h1 + h2) / ((h0 + h1) * (h0 + h1 + h2));
        const double w2 = -h0 * h1 / ((h0 + h1 + h2) * (h1 + h2));
        const double w1 = 1.0 - w0 - w2;
        aj[j] = u == 1 ? w0 : w1;
        cp[j] = u == 1 ? w1 : w0;
        c2[j] = w2;
      }
    }
  }
  __syncwarp();

  for (int f = 0; f < a.nfield; ++f) {
    __syncthreads();  // every warp is done with the field before, whose slot is refilled now
    issue(f + SLOTS - 1);
    pending<SLOTS - 1>();
    __syncthreads();  // the field is in its slot
    const double* Q = ring + ((f % SLOTS) * COLS + warp) * RP;
    double* q2 = a.q_out + qo + f * a.sQqo;
    // w[i]: mean of layer u0 - 2 + i (clamped into the column); D[i] the jump w[i+1] - w[i]
    double w[NPL + 4], D[NPL + 3];
#pragma unroll
    for (int i = 0; i < NPL + 4; ++i) w[i] = Q[pd(min(max(u0 - 2 + i, 0), km - 1))];
#pragma unroll
    for (int i = 0; i < NPL + 3; ++i) D[i] = w[i + 1] - w[i];
    bool gen = odd;
#pragma unroll
    for (int j = 0; j < NPL; ++j) gen |= huge_or_nan(w[j + 2]);
    gen = __any_sync(FULL, gen);
    if (gen && lane == (f & 31)) general |= 1u << (f >> 5);
    // -------------------------------------------- interface values a[0..km]
    double st[NPL], dm[NPL];
#pragma unroll
    for (int j = 0; j < NPL; ++j) dm[j] = 0.0;
    if (km == 1) {
#pragma unroll
      for (int j = 0; j < NPL; ++j) st[j] = w[2];
    } else if (KORD == 9) {
      double r[NPL], be = 0.0, y[NPL];
#pragma unroll
      for (int j = 0; j < NPL; ++j) {
        const int u = u0 + j;
        const double qa = u == 0 ? w[j + 2] : w[j + 1];
        const double qb = u == 0 ? w[j + 3] : (u == km ? w[j] : w[j + 2]);
        r[j] = fma(e1[j], qa, e2[j] * qb);
        if (a.iv == -2 && u == km) r[j] = qsv;  // the given surface value (aj is 0 there)
        be = j == 0 ? r[j] : fma(aj[j], be, r[j]);
      }
#pragma unroll
      for (int o = 1, s = 0; o < 32; o <<= 1, ++s) {
        const double p = __shfl_up_sync(FULL, be, o);
        const double v = fma(mf[s], p, be);
        be = lane >= o ? v : be;
      }
      double yp = __shfl_up_sync(FULL, be, 1);
#pragma unroll
      for (int j = 0; j < NPL; ++j) {
        y[j] = yp = (u0 + j == 0) ? r[j] : fma(aj[j], yp, r[j]);
      }
      be = y[NPL - 1];
#pragma unroll
      for (int j = NPL - 2; j >= 0; --j) be = fma(negv(cp[j]), be, y[j]);
#pragma unroll
      for (int o = 1, s = 0; o < 32; o <<= 1, ++s) {
        const double p = __shfl_down_sync(FULL, be, o);
        const double v = fma(mb[s], p, be);
        be = lane + o < 32 ? v : be;
      }
      double av = __shfl_down_sync(FULL, be, 1);
      if (lane == 31) av = 0.0;
#pragma unroll
      for (int j = NPL - 1; j >= 0; --j) {
        const int u = u0 + j;
        av = u < km ? fma(negv(cp[j]), av, y[j]) : y[j];
        const double dc = D[j + 1], dl = u > 1 ? D[j] : dc, dr = u < km - 1 ? D[j + 2] : dc;
        // the end interfaces: into the range of the two outermost layers
        const double qa = u == 0 ? w[j + 2] : u >= km ? w[j] : w[j + 1];
        const double qb = u == 0 ? w[j + 3] : u >= km ? w[j + 1] : w[j + 2];
        const bool end = u == 0 || u >= km;
        const double v = limit9(av, qa, qb, end ? 1.0 : dl, end ? 1.0 : dr, a.iv, floor_v);
        st[j] = u >= km && a.iv == -2 ? av : v;
      }
    } else {
      // slopes of the lane's layers, limited by the range of the layer and its neighbours
#pragma unroll
      for (int j = 0; j < NPL; ++j) {
        const double dq = fma(e1[j], D[j + 2], e2[j] * D[j + 1]);
        const bool mono = (__double2hiint(D[j + 1]) ^ __double2hiint(D[j + 2])) >= 0;
        const double m = mag_min(scale2<-1>(absv(dq)), mag_min(absv(D[j + 1]), absv(D[j + 2])));
        const int u = u0 + j;
        dm[j] = mono && u >= 1 && u <= km - 2 ? signed_as(m, dq) : 0.0;
      }
      const double dmw = __shfl_up_sync(FULL, dm[NPL - 1], 1);
      double last = 0.0;
#pragma unroll
      for (int j = 0; j < NPL; ++j) {
        const int u = u0 + j;
        const bool inner = u >= 2 && u <= km - 2;
        const double qa = w[j + 1], qb = w[j + 2], q3 = u == 1 ? w[j + 3] : w[j];
        const double x0 = inner ? fma(aj[j], D[j + 1], qa) : aj[j] * qa;
        const double x1 = fma(cp[j], inner ? (j ? dm[j ? j - 1 : 0] : dmw) : qb, x0);
        const double x2 = fma(inner ? negv(c2[j]) : c2[j], inner ? dm[j] : q3, x1);
        const bool upw = less(qa, qb);
        const double lo = upw ? qa : qb, hi = upw ? qb : qa;
        const double cl = less(x2, lo) ? lo : less(hi, x2) ? hi : x2;
        st[j] = inner ? x2 : cl;
      }
      // the outermost interfaces from the next ones
      last = __shfl_up_sync(FULL, st[NPL - 1], 1);
      if (lane == 0) st[0] = 2.0 * w[2] - st[1];
#pragma unroll
      for (int j = 0; j < NPL; ++j)
        if (u0 + j == km) st[j] = a.iv == -2 ? qsv : 2.0 * w[j + 1] - (j ? st[j ? j - 1 : 0] : last);
    }
    const double st_end = __shfl_down_sync(FULL, st[0], 1);
    // ------------------------------------------ sub-grid parabolas of layers
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
      const int u = u0 + j;
      const double qk = w[j + 2];
      double bl = st[j] - qk, br = (j + 1 < NPL ? st[j + 1 < NPL ? j + 1 : 0] : st_end) - qk;
      if (km == 1) bl = br = 0.0;
      const bool end = u < 2 || u > km - 3;
      if (KORD == 9) {
        const double D0 = D[j + 1], D1 = D[j + 2];
        const bool flat = opp(D0, D1) && (opp(D[j], D0) || opp(D1, D[j + 3]));
        const bool nonmono = mag_less(absv(br - bl), absv(3.0 * (bl + br)));
        const double pr = scale2<1>(D0), lr = fma(-1.5, D[j], pr);
        const double pl = negv(scale2<1>(D1)), ll = fma(1.5, D[j + 3], pl);
        const double brc = clamp0(br, pr, lr), blc = clamp0(bl, pl, ll);
        if (!end) {
          bl = flat ? 0.0 : (nonmono ? blc : bl);
          br = flat ? 0.0 : (nonmono ? brc : br);
        }
      } else if (!end) {
        const double ax = absv(scale2<1>(dm[j]));
        const double ml = mag_min(ax, absv(bl)), mr = mag_min(ax, absv(br));
        bl = neg(dm[j]) ? ml : negv(ml);
        br = neg(dm[j]) ? negv(mr) : mr;
      }
      if (end) {  // CW84 eq. 1.10 on the two layers at each end
        const double d = br - bl, t = 3.0 * d * (bl + br), d2 = d * d;
        const bool big = mag_less(d2, absv(t)), lo = big && neg(t), hi = big && !lo;
        const double nl = lo ? negv(scale2<1>(br)) : bl, nr = hi ? negv(scale2<1>(bl)) : br;
        const bool flat = !opp(bl, br);
        bl = flat ? 0.0 : nl;
        br = flat ? 0.0 : nr;
      }
      double s = bl + br, da = br - bl, pl = qk + bl;
      if (a.iv >= 0) {
        // minimum of the parabola: an edge, or q - s/4 - da^2/(12 s) >= q - s inside (s > |da| / 3); it can
        // lie below the floor only where an edge does or s exceeds the mean's height above the floor
        const double qf = floor_v == 0.0 ? qk : qk - floor_v;
        const bool low_edge = less(pl, floor_v) || less(qk + br, floor_v);
        if (low_edge || (pos(s) && less(qf, s))) {
          // inside, the minimum lies below the floor where 3 s^2 + da^2 > 12 s (q - floor)
          const double s3 = 3.0 * s, da2 = da * da;
          const bool inner = pos(s) && mag_less(absv(da), s3);
          if (low_edge || (inner && less(12.0 * s * qf, fma(s3, s, da2)))) {
            const double pr = qk + br;
            double pmin = less(pl, pr) ? pl : pr;
            if (inner) {
              const double in = (qk - scale2<-2>(s)) - da2 * fast_rcp(12.0 * s);
              pmin = less(in, pmin) ? in : pmin;
            }
            const double lam = pos(qf) ? fast_div(qf, qk - pmin) : 0.0;
            bl *= lam;
            br *= lam;
            s = bl + br;
            da = br - bl;
            pl = qk + bl;
          }
        }
      }
      if (u < km) {
        const int i = pd(u);
        S.l[i] = pl;
        S.h[i] = fma(-1.5, s, scale2<-1>(da));
        S.s[i] = s;
      }
    }
    __syncwarp();
    // ------------------------------------------------------- target layers
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
      const int t = u0 + j;
      if (t < kn) {
        const unsigned sc = sched[j];
        const int i = pd(t), it = pd(sc & 0xff), ib = pd((sc >> 8) & 0xff);
        const double vt = (sc >> 16) & 1 ? Q[it] : S.l[it], vb = (sc >> 17) & 1 ? Q[ib] : S.l[ib];
        const double mt = fma(S.S1[i], S.h[it], fma(S.Q1[i], S.s[it], vt));
        const double mb_ = fma(S.S2[i], S.h[ib], fma(S.Q2[i], S.s[ib], vb));
        double out = fma(S.w2[i], mb_, S.w1[i] * mt);
        if ((sc >> 18) & 1) {
          double mass = 0.0;
          for (int m = (int)(sc & 0xff) + 1; m < (int)((sc >> 8) & 0xff); ++m) mass = fma(Q[pd(m)], S.dp[pd(m)], mass);
          out = fma(mass, rdpk_of(t), out);
        }
        if (real && !gen) q2[(long long)t * a.sQk] = out;
      }
    }
  }
  if (__any_sync(FULL, general != 0))
    general_fields<KORD, NPL>(S, ring + warp * RP, general, qo, col, lane, real, a);
}

template <int KORD, int NPL>
cudaError_t launch64(const RemapArgs<double>& a, cudaStream_t s) {
  RemapArgs<double> b = a;
  for (int f = 0; f < a.nfield; f += MAX_FIELDS) {
    b.nfield = std::min(MAX_FIELDS, a.nfield - f);
    b.q_in = a.q_in + f * a.sQq;
    b.q_out = a.q_out + f * a.sQqo;
    k_remap64<KORD, NPL><<<(unsigned)((a.ncol + COLS - 1) / COLS), 32 * COLS, smem64<NPL>(), s>>>(b);
  }
  return cudaGetLastError();
}

template <int KORD, int NPL>
cudaError_t allow() {
  return cudaFuncSetAttribute(k_remap64<KORD, NPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem64<NPL>());
}

}  // namespace

// Raise the kernels' dynamic shared-memory limit (prepare_remap_kernels calls it once, before any capture).
cudaError_t prepare_remap64() {
  const cudaError_t es[] = {allow<9, 2>(), allow<9, 3>(), allow<9, 4>(), allow<9, 5>(),
                            allow<4, 2>(), allow<4, 3>(), allow<4, 4>(), allow<4, 5>()};
  for (cudaError_t e : es)
    if (e != cudaSuccess) return e;
  return cudaSuccess;
}

// FP64 columns, kord 9 or 4, km and kn up to KMAX.  A lane owns the fewest layers
// (2 to 5) with which the 32 lanes hold all km + 1 interfaces: idle lanes cost the
// FP64 pipe what busy ones do.
cudaError_t launch_remap64(const RemapArgs<double>& a, int kord, cudaStream_t s) {
  const int npl = std::max(2, std::max(a.km, a.kn) / 32 + 1);
  if (kord == 9)
    return npl == 2 ? launch64<9, 2>(a, s) : npl == 3 ? launch64<9, 3>(a, s) : npl == 4 ? launch64<9, 4>(a, s)
                                                                                          : launch64<9, 5>(a, s);
  return npl == 2 ? launch64<4, 2>(a, s) : npl == 3 ? launch64<4, 3>(a, s) : npl == 4 ? launch64<4, 4>(a, s)
                                                                                        : launch64<4, 5>(a, s);
}

}  // namespace fv3g
