// fv3g_adjoint.cu -- the linearised transport step (fv3g_adjoint.cuh): face
// weights of the PPM sweeps on the trajectory, the tangent-linear substep,
// the hand-written adjoint substep (transposed gathers, corner and halo
// transposes) and the reverse sweep of the kord-4 column remap.
#include <algorithm>

#include "fv3g_adjoint.cuh"
#include "fv3g_dual.cuh"
#include "fv3g_fp64.cuh"
#include "fv3g_profile.cuh"
#include "fv3g_remap.cuh"
#include "fv3g_stencil.cuh"

namespace fv3g {
namespace {

using D2 = Dual<double>;

// one-sided interface weights at cube-face edges (Putman & Lin 2007)
constexpr double kS11 = 11.0 / 14.0, kS14 = 4.0 / 7.0, kS15 = 3.0 / 14.0;  // hord 8
constexpr double kC1 = -2.0 / 14.0, kC2 = 11.0 / 14.0, kC3 = 5.0 / 14.0;   // hord 1 / 5

// ------------------------------------------------------- face-local PPM ---
// Flux through face f (between cells f-1 and f) of one line, read through
// X(m) for the cells m = f-3..f+2 it depends on, with the cell widths DX(m)
// along the line (one-sided edge values) and the face's Courant number c.
// eLo / eHi: the line's cube-face edge faces (tile interior above eLo, below
// eHi) or NO_EDGE.  The same scheme as the substep kernel's lines:
//   hord 8: monotonized central slopes, interfaces from them, the Lin (2004)
//           limit of the edge deviations; at a cube-face edge the edge value
//           (mean of the two one-sided extrapolations) clamped to the two
//           cells beside it, the next interfaces inward one-sided, the one
//           beyond unlimited, then CW84 on the three edge cells;
//   hord 1 / 5: fourth-order interfaces, one-sided three-cell interfaces
//           beside a cube-face edge and the unlimited edge value; the face
//           takes the first-order upwind value unless a cell beside it
//           passes bl br < 0 (hord 5) or |lim_fac (bl + br)| < |bl - br|
//           (hord 1).
template <typename T, class XF, class DF>
__device__ T ppm_face(int hord, double lim_fac, int f, const XF& X, const DF& DX, double c, int eLo, int eHi) {
  auto edge_mean = [&](int e) -> T {
    const T d2 = T(DX(e - 2)), d1 = T(DX(e - 1)), d0 = T(DX(e)), d3 = T(DX(e + 1));
    const T xl = ((T(2) * d1 + d2) * X(e - 1) - d1 * X(e - 2)) / (d2 + d1);
    const T xr = ((T(2) * d0 + d3) * X(e) - d0 * X(e + 1)) / (d0 + d3);
    return T(0.5) * (xl + xr);
  };
  auto in = [f](int m) { return m == f - 1 || m == f; };
  T bl[2], br[2];  // deviations of cells f-1 and f
  bool smt[2] = {true, true};
  if (hord == 8) {
    // the forms of the substep kernel, so that exact ties (flat lines) take
    // its one-sided derivatives: its line march (clamped slopes, copysign)
    // away from cube-face edges, the generic cell values of its edge windows
    // (cells e-2 .. e+1 of an edge e) beside them
    auto DM = [&](int m) -> T { return vl_slope(X(m - 1), X(m), X(m + 1)); };
    auto AL = [&](int g) -> T { return T(0.5) * (X(g - 1) + X(g)) + (DM(g - 1) - DM(g)) * T(1.0 / 3.0); };
    auto DMC = [&](int m) -> T {
      const T xm = X(m - 1), x0 = X(m), xp = X(m + 1);
      const T xt = T(0.25) * (xp - xm);
      return copysign_t(tmin3(tabs(xt), tmax3(xm, x0, xp) - x0, x0 - tmin3(xm, x0, xp)), xt);
    };
    auto ALC = [&](int g) -> T { return T(0.5) * (X(g - 1) + X(g)) + (DMC(g - 1) - DMC(g)) * T(1.0 / 3.0); };
    auto window = [&](int m) {
      return (eLo != NO_EDGE && m >= eLo - 2 && m <= eLo + 1) || (eHi != NO_EDGE && m >= eHi - 2 && m <= eHi + 1);
    };
    for (int h = 0; h < 2; ++h) {
      const int m = f - 1 + h;
      if (window(m)) {
        const T xt = T(2) * DM(m);
        bl[h] = -tsign(tmin(tabs(xt), tabs(AL(m) - X(m))), xt);
        br[h] = tsign(tmin(tabs(xt), tabs(AL(m + 1) - X(m))), xt);
      } else {
        const T dmm = DMC(m);
        const T xt = dmm + dmm;
        const T axt = tabs(xt);
        bl[h] = copysign_t(tmin(axt, tabs(ALC(m) - X(m))), -xt);
        br[h] = copysign_t(tmin(axt, tabs(ALC(m + 1) - X(m))), xt);
      }
    }
    auto setl = [&](int m, T v) { if (in(m)) bl[m - f + 1] = v; };
    auto setr = [&](int m, T v) { if (in(m)) br[m - f + 1] = v; };
    auto cw = [&](int m) { if (in(m)) cw84(bl[m - f + 1], br[m - f + 1]); };
    if (eLo != NO_EDGE) {
      const int e = eLo;
      const bool cL = in(e - 1), c0 = in(e), cR = in(e + 1);
      if (cL || c0 || cR) {
        T a0 = T(0), ap = T(0);
        if (cL || c0) a0 = clamp2(edge_mean(e), X(e - 1), X(e));
        if (c0 || cR) ap = T(kS15) * X(e) + T(kS11) * X(e + 1) - T(kS14) * DM(e + 1);
        if (cL) {
          setl(e - 1, T(kS14) * DM(e - 2) + T(kS11) * (X(e - 2) - X(e - 1)));
          setr(e - 1, a0 - X(e - 1));
        }
        if (c0) {
          setl(e, a0 - X(e));
          setr(e, ap - X(e));
        }
        if (cR) {
          setl(e + 1, ap - X(e + 1));
          setr(e + 1, AL(e + 2) - X(e + 1));
        }
        cw(e - 1);
        cw(e);
        cw(e + 1);
      }
    }
    if (eHi != NO_EDGE) {
      const int e = eHi;
      const bool cL2 = in(e - 2), cL = in(e - 1), c0 = in(e);
      if (cL2 || cL || c0) {
        T am = T(0), a0 = T(0);
        if (cL2 || cL) am = T(kS15) * X(e - 1) + T(kS11) * X(e - 2) + T(kS14) * DM(e - 2);
        if (cL || c0) a0 = clamp2(edge_mean(e), X(e - 1), X(e));
        if (cL2) {
          setl(e - 2, AL(e - 2) - X(e - 2));
          setr(e - 2, am - X(e - 2));
        }
        if (cL) {
          setl(e - 1, am - X(e - 1));
          setr(e - 1, a0 - X(e - 1));
        }
        if (c0) {
          setl(e, a0 - X(e));
          setr(e, T(kS11) * (X(e + 1) - X(e)) - T(kS14) * DM(e + 1));
        }
        cw(e - 2);
        cw(e - 1);
        cw(e);
      }
    }
  } else {
    auto AL = [&](int g) -> T {
      for (int side = 1; side >= 0; --side) {  // the high edge's one-sided values take precedence
        const int e = side ? eHi : eLo;
        if (e == NO_EDGE) continue;
        if (g == e - 1) return T(kC1) * X(e - 3) + T(kC2) * X(e - 2) + T(kC3) * X(e - 1);
        if (g == e) return edge_mean(e);
        if (g == e + 1) return T(kC3) * X(e) + T(kC2) * X(e + 1) + T(kC1) * X(e + 2);
      }
      return T(7.0 / 12.0) * (X(g - 1) + X(g)) - T(1.0 / 12.0) * (X(g - 2) + X(g + 1));
    };
    for (int h = 0; h < 2; ++h) {
      const int m = f - 1 + h;
      bl[h] = AL(m) - X(m);
      br[h] = AL(m + 1) - X(m);
      if (hord == 5) smt[h] = value_of(bl[h]) * value_of(br[h]) < 0.0;
      else smt[h] = fabs(lim_fac * value_of(bl[h] + br[h])) < fabs(value_of(bl[h] - br[h]));
    }
  }
  const bool high = hord == 8 || smt[0] || smt[1];
  const double ac = fabs(c), w1 = 1.0 - ac, w2 = ac * w1;
  if (c > 0.0) return high ? (X(f - 1) + T(w1) * br[0]) - T(w2) * (bl[0] + br[0]) : X(f - 1);
  return high ? (X(f) + T(w1) * bl[1]) - T(w2) * (bl[1] + br[1]) : X(f);
}

// Faces whose cells f-1 or f take a one-sided value at a cube-face edge e
// (cells e-2 .. e+1 do), in the sweeps' lines.
__device__ __forceinline__ bool edge_face(int f, int eLo, int eHi) {
  return (eLo != NO_EDGE && f >= eLo - 2 && f <= eLo + 2) || (eHi != NO_EDGE && f >= eHi - 2 && f <= eHi + 2);
}

// The six weights of face f's flux on cells f-3..f+2 and the flux value, away
// from cube-face edges, in closed form: the flux reads the upwind cell m, its
// deviations bl, br and (hord 1, 5) the filter tests of both cells, and every
// branch leaves a linear form of the means, so one evaluation of the values
// and about twenty multiply-adds replace a forward-mode pass per cell.  FP64
// runs at 1/64 of the FP32 rate, so the count of FP64 operations is the cost:
// six C96 tiles x 64 levels x 4 tracers, hord 5, six substeps took 505 ms in
// both kernels with six passes per face.  The branch conventions are those of
// ppm_face on dual numbers (on a tie the later operand); faces with an infinity or a NaN in their
// window are reported in odd and left to k_lin_odd.
__device__ __forceinline__ void put_weights(double* w, long long ws, const double* W) {
#pragma unroll
  for (int s = 0; s < 6; ++s) w[s * ws] = W[s];
}

__device__ __forceinline__ bool odd_window(const double* x, double c) {
  bool odd = inf_or_nan(c);
#pragma unroll
  for (int s = 0; s < 6; ++s) odd |= inf_or_nan(x[s]);
  return odd;
}

// Slope of the middle cell of (xm, x0, xp) and its derivatives p on the three.
// Every comparison is a sign of one of three differences.
__device__ __forceinline__ double slope_grad(double xm, double x0, double xp, double* p) {
  const double dm = x0 - xm, dp = xp - x0, s = xp - xm;
  const double ax = scale2<-2>(absv(s));
  const bool hi_m = neg(dm) && neg(s), hi_0 = !neg(dm) && neg(dp);  // the largest: xm, x0, else xp
  const bool lo_m = pos(dm) && pos(s), lo_0 = !pos(dm) && pos(dp);  // the smallest
  const double up = hi_m ? negv(dm) : hi_0 ? 0.0 : dp, dn = lo_m ? dm : lo_0 ? 0.0 : absv(dp);
  const bool lim = mag_less(ax, up);
  const double m1 = lim ? ax : up;
  const bool use_dn = !mag_less(m1, dn), use_up = !use_dn && !lim;
  const double mag = absv(use_dn ? dn : m1);
  const bool ng = __double2hiint(s) < 0;
  const double sg = ng ? -1.0 : 1.0;
  p[0] = use_dn ? (lo_m ? negv(sg) : 0.0) : use_up ? (hi_m ? sg : 0.0) : -0.25;
  p[1] = use_dn ? (lo_0 ? 0.0 : sg) : use_up ? (hi_0 ? 0.0 : negv(sg)) : 0.0;
  p[2] = use_dn ? ((lo_m || lo_0) ? 0.0 : negv(sg)) : use_up ? ((hi_m || hi_0) ? 0.0 : sg) : 0.25;
  return signed_as(mag, s);
}

template <class XV>
__device__ __forceinline__ double face_weights(int hord, double lim_fac, int f, const XV& xv, double c, double* w,
                                               long long ws, int* odd) {
  double x[6], W[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int s = 0; s < 6; ++s) x[s] = xv(f - 3 + s);
  if (odd_window(x, c)) *odd = 1;
  const bool left = pos(c);  // upwind cell f-1 (window cell 2), else f (window cell 3)
  const double ac = absv(c), w1 = 1.0 - ac, w2 = ac * w1;
  const double wd = w1 - w2, nw2 = negv(w2);
  const double cl = left ? nw2 : wd, cr = left ? wd : nw2;  // flux = x_m + cl bl + cr br
  if (hord == 8) {
    double y[5], p0[3], p1[3], p2[3], V[5];  // cells m-2 .. m+2
#pragma unroll
    for (int s = 0; s < 5; ++s) y[s] = left ? x[s] : x[s + 1];
    const double d0 = slope_grad(y[0], y[1], y[2], p0), d1 = slope_grad(y[1], y[2], y[3], p1),
                 d2 = slope_grad(y[2], y[3], y[4], p2);
    const double axt = scale2<1>(absv(d1));  // |2 dm|; d1 has the sign of the slope
    const double tl = (0.5 * (y[1] + y[2]) + (d0 - d1) * (1.0 / 3.0)) - y[2];
    const double tr = (0.5 * (y[2] + y[3]) + (d1 - d2) * (1.0 / 3.0)) - y[2];
    const bool lim_l = mag_less(axt, absv(tl)), lim_r = mag_less(axt, absv(tr));
    const double bl = negv(signed_as(lim_l ? axt : absv(tl), d1)), br = signed_as(lim_r ? axt : absv(tr), d1);
    // derivatives of bl: -2 dm where limited, else those of +-tl; br likewise
    const double kl = (__double2hiint(tl) ^ __double2hiint(d1)) < 0 ? cl : negv(cl);
    const double kr = (__double2hiint(tr) ^ __double2hiint(d1)) < 0 ? negv(cr) : cr;
    const double hl = lim_l ? 0.0 : 0.5 * kl, hr = lim_r ? 0.0 : 0.5 * kr;
    const double gl = lim_l ? 0.0 : kl * (1.0 / 3.0), gr = lim_r ? 0.0 : kr * (1.0 / 3.0);
    const double g1 = (lim_l ? -2.0 * cl : negv(gl)) + (lim_r ? 2.0 * cr : gr);
    V[0] = gl * p0[0];
    V[1] = hl + gl * p0[1] + g1 * p1[0];
    V[2] = (1.0 - hl - hr) + gl * p0[2] + g1 * p1[1] - gr * p2[0];
    V[3] = hr + g1 * p1[2] - gr * p2[1];
    V[4] = -gr * p2[2];
#pragma unroll
    for (int s = 0; s < 6; ++s) W[s] = left ? (s < 5 ? V[s] : 0.0) : (s > 0 ? V[s - 1] : 0.0);
    put_weights(w, ws, W);
    return (y[2] + w1 * (left ? br : bl)) - w2 * (bl + br);
  }
  double al[3], bl[2], br[2];
#pragma unroll
  for (int g = 0; g < 3; ++g) al[g] = (7.0 / 12.0) * (x[g + 1] + x[g + 2]) - (1.0 / 12.0) * (x[g] + x[g + 3]);
  bool high = false;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    bl[h] = al[h] - x[h + 2];
    br[h] = al[h + 1] - x[h + 2];
    if (hord == 5) high = high || opp(bl[h], br[h]);
    else high = high || fabs(lim_fac * (bl[h] + br[h])) < fabs(bl[h] - br[h]);
  }
  const double xu = left ? x[2] : x[3];
  const double a = high ? cl : 0.0, b = high ? cr : 0.0;
  const double va = (-1.0 / 12.0) * a, vb = (-1.0 / 12.0) * b;
  const double V[5] = {va, fma(7.0 / 12.0, a, vb), fma(-5.0 / 12.0, a + b, 1.0), fma(7.0 / 12.0, b, va), vb};
#pragma unroll
  for (int s = 0; s < 6; ++s) W[s] = left ? (s < 5 ? V[s] : 0.0) : (s > 0 ? V[s - 1] : 0.0);
  put_weights(w, ws, W);
  const double bu = left ? bl[0] : bl[1], ru = left ? br[0] : br[1];
  return high ? (xu + w1 * (left ? ru : bu)) - w2 * (bu + ru) : xu;
}

// The same beside a cube-face edge.  hord 1 / 5: the interfaces' taps, the
// one-sided ones included.  hord 8: one forward-mode pass of ppm_face per
// cell (six faces of a line).
template <class XV, class DF>
__device__ __forceinline__ double forward_weights(int hord, double lim_fac, int f, const XV& xv, const DF& DX, double c,
                                                  int eLo, int eHi, double* w, long long ws) {
  double val = 0.0;
#pragma unroll 1
  for (int s = 0; s < 6; ++s) {
    const int ms = f - 3 + s;
    auto X = [&](int m) -> D2 { return D2(xv(m), m == ms ? 1.0 : 0.0); };
    const D2 r = ppm_face<D2>(hord, lim_fac, f, X, DX, c, eLo, eHi);
    w[s * ws] = r.d;
    val = r.v;
  }
  return val;
}
template <class XV, class DF>
__device__ double edge_face_weights(int hord, double lim_fac, int f, const XV& xv, const DF& DX, double c, int eLo,
                                    int eHi, double* w, long long ws, int* odd) {
  if (hord == 8) return forward_weights(hord, lim_fac, f, xv, DX, c, eLo, eHi, w, ws);
  double x[6];
#pragma unroll
  for (int s = 0; s < 6; ++s) x[s] = xv(f - 3 + s);
  if (odd_window(x, c)) *odd = 1;
  double G[3][6], al[3];  // taps on the window and values of interfaces f-1, f, f+1
#pragma unroll
  for (int g = 0; g < 3; ++g) {
    const int u = f - 1 + g;
    double t[4] = {-1.0 / 12.0, 7.0 / 12.0, 7.0 / 12.0, -1.0 / 12.0};
    int base = u - 2;
    for (int side = 0; side < 2; ++side) {  // the high edge's one-sided values take precedence
      const int e = side ? eHi : eLo;
      if (e == NO_EDGE) continue;
      if (u == e - 1) {
        base = e - 3;
        t[0] = kC1; t[1] = kC2; t[2] = kC3; t[3] = 0.0;
      } else if (u == e) {
        base = e - 2;
        const double d2 = DX(e - 2), d1 = DX(e - 1), d0 = DX(e), d3 = DX(e + 1);
        t[0] = -0.5 * d1 / (d2 + d1);
        t[1] = 0.5 * (2.0 * d1 + d2) / (d2 + d1);
        t[2] = 0.5 * (2.0 * d0 + d3) / (d0 + d3);
        t[3] = -0.5 * d0 / (d0 + d3);
      } else if (u == e + 1) {
        base = e;
        t[0] = kC3; t[1] = kC2; t[2] = kC1; t[3] = 0.0;
      }
    }
    al[g] = 0.0;
#pragma unroll
    for (int s = 0; s < 6; ++s) {
      const int k = f - 3 + s - base;
      G[g][s] = k == 0 ? t[0] : k == 1 ? t[1] : k == 2 ? t[2] : k == 3 ? t[3] : 0.0;
      al[g] += G[g][s] * x[s];
    }
  }
  bool high = false;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const double bl = al[h] - x[h + 2], br = al[h + 1] - x[h + 2];
    high = high || (hord == 5 ? bl * br < 0.0 : fabs(lim_fac * (bl + br)) < fabs(bl - br));
  }
  const bool left = c > 0.0;
  const double ac = fabs(c), w1 = 1.0 - ac, w2 = ac * w1;
  const double a = high ? (left ? -w2 : w1 - w2) : 0.0, b = high ? (left ? w1 - w2 : -w2) : 0.0;
  const double xu = left ? x[2] : x[3];
#pragma unroll
  for (int s = 0; s < 6; ++s) {
    const double Ga = left ? G[0][s] : G[1][s], Gb = left ? G[1][s] : G[2][s];
    const bool up = s == (left ? 2 : 3);
    w[s * ws] = a * Ga + b * Gb + (up ? (1.0 - a) - b : 0.0);
  }
  const double bl = (left ? al[0] : al[1]) - xu, br = (left ? al[1] : al[2]) - xu;
  return high ? (xu + w1 * (left ? br : bl)) - w2 * (bl + br) : xu;
}

// ------------------------------------------------------- plane indexing ---
struct Cell {
  int pl, t, k;  // plane, tile, level
  int i, j;      // tile indices
  long long p;   // offset in the plane
  long long q0, lev, met;  // plane offsets: q-shaped arrays, per-level fields, metrics
};

__device__ __forceinline__ bool cell_of(const LinArgs& a, Cell& c) {
  c.p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c.p >= a.P) return false;
  c.pl = blockIdx.y;
  c.i = a.pg.isd + (int)(c.p % a.pg.pitch);
  c.j = a.pg.jsd + (int)(c.p / a.pg.pitch);
  if (c.i > a.ied || c.j > a.jed) return false;  // plane padding: never read
  const int per_tile = a.nq * a.npz;
  c.t = c.pl / per_tile;
  c.k = c.pl % a.npz;
  c.q0 = (long long)c.pl * a.P;
  c.lev = ((long long)c.t * a.npz + c.k) * a.P;
  c.met = (long long)c.t * a.P;
  return true;
}

__device__ __forceinline__ bool in_rng(int v, int lo, int hi) { return v >= lo && v <= hi; }
__device__ __forceinline__ bool inside_data(const LinArgs& a, int i, int j) {
  return in_rng(i, a.isd, a.ied) && in_rng(j, a.jsd, a.jed);
}
// a cell of a copy_corners block that the sweeps fill
__device__ __forceinline__ bool corner_cell(const LinArgs& a, int i, int j) {
  const bool oi = i < 1 || i > a.npx - 1, oj = j < 1 || j > a.npy - 1;
  if (!(oi && oj)) return false;
  const int bit = (i < 1 ? 0 : 1) + (j < 1 ? 0 : 2);
  return (a.corners >> bit) & 1;
}

__device__ __forceinline__ double ra_y(const LinArgs& a, const Cell& c, int i, int j) {
  const PlaneGeom& pg = a.pg;
  if (a.ra_y) return a.ra_y[c.lev + pg.at(i, j)];
  return a.area[c.met + pg.at(i, j)] + a.yfx[c.lev + pg.at(i, j)] - a.yfx[c.lev + pg.at(i, j + 1)];
}
__device__ __forceinline__ double ra_x(const LinArgs& a, const Cell& c, int i, int j) {
  const PlaneGeom& pg = a.pg;
  if (a.ra_x) return a.ra_x[c.lev + pg.at(i, j)];
  return a.area[c.met + pg.at(i, j)] + a.xfx[c.lev + pg.at(i, j)] - a.xfx[c.lev + pg.at(i + 1, j)];
}

__device__ __forceinline__ double inv_ra_y(const LinArgs& a, const Cell& c, int i, int j) {
  return a.rry ? a.rry[c.lev + a.pg.at(i, j)] : fast_rcp(ra_y(a, c, i, j));
}
__device__ __forceinline__ double inv_ra_x(const LinArgs& a, const Cell& c, int i, int j) {
  return a.rrx ? a.rrx[c.lev + a.pg.at(i, j)] : fast_rcp(ra_x(a, c, i, j));
}

// face ranges of the four sweeps
__device__ __forceinline__ bool yi_face(const LinArgs& a, int i, int j) {  // inner y: every column
  return in_rng(j, a.js, a.je + 1) && in_rng(i, a.isd, a.ied);
}
__device__ __forceinline__ bool xi_face(const LinArgs& a, int i, int j) {  // inner x: every row
  return in_rng(i, a.is, a.ie + 1) && in_rng(j, a.jsd, a.jed);
}
__device__ __forceinline__ bool xo_face(const LinArgs& a, int i, int j) {  // outer x: compute rows
  return in_rng(i, a.is, a.ie + 1) && in_rng(j, a.js, a.je);
}
__device__ __forceinline__ bool yo_face(const LinArgs& a, int i, int j) {  // outer y: compute columns
  return in_rng(j, a.js, a.je + 1) && in_rng(i, a.is, a.ie);
}

// ---------------------------------------------------------- trajectory ---
// Level-only factors of a substep, shared by its tracers: dp1/dp2 and rarea/dp2
// on the compute cells.  An IEEE division is about eleven FP64 instructions: with these
// and the forward substeps' 1/ra_x and 1/ra_y, a substep's k_ad_mid, k_ad_faces, k_ad_inner
// and k_lin_mid take 0.24, 0.30, 0.54 and 0.25 ms (1.62, 1.15, 1.07, 0.72 ms dividing; six
// C96 tiles x 64 levels x 4 tracers).
__global__ void k_lin_ratios(const LinArgs a) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= a.P) return;
  const int i = a.pg.isd + (int)(p % a.pg.pitch), j = a.pg.jsd + (int)(p / a.pg.pitch);
  if (!in_rng(i, a.is, a.ie) || !in_rng(j, a.js, a.je)) return;
  const long long lev = (long long)blockIdx.y * a.P + p, met = (long long)(blockIdx.y / a.npz) * a.P + p;
  const double r = fast_rcp(a.dp2[lev]);
  a.dr[lev] = a.dp1[lev] * r;
  a.r2[lev] = a.rarea[met] * r;
}

// The two corner-filled copies of the halo-filled input (copy_corners for x
// and for y sweeps).
__global__ void k_lin_corners(const LinArgs a, const double* q, double* c1, double* c2) {
  Cell c;
  if (!cell_of(a, c)) return;
  const double* qp = q + c.q0;
  if (corner_cell(a, c.i, c.j)) {
    int i1 = c.i, j1 = c.j, i2 = c.i, j2 = c.j;
    corner_rotate(i1, j1, a.npx, a.npy, 1);
    corner_rotate(i2, j2, a.npx, a.npy, 2);
    c1[c.q0 + c.p] = inside_data(a, i1, j1) ? qp[a.pg.at(i1, j1)] : 0.0;
    c2[c.q0 + c.p] = inside_data(a, i2, j2) ? qp[a.pg.at(i2, j2)] : 0.0;
  } else {
    c1[c.q0 + c.p] = qp[c.p];
    c2[c.q0 + c.p] = qp[c.p];
  }
}

// Inner sweeps: y faces for every column of the data domain on the dir-2
// copy, x faces for every row on the dir-1 copy: weights and flux values.
// Faces beside a cube-face edge are left to k_lin_edges.
__global__ void k_lin_inner(const LinArgs a, const LinTraj tr) {
  Cell c;
  if (!cell_of(a, c)) return;
  const long long ws = (long long)a.nt * a.nq * a.npz * a.P;
  const PlaneGeom& pg = a.pg;
  if (!yi_face(a, c.i, c.j)) {
    for (int s = 0; s < 6; ++s) tr.wyi[s * ws + c.q0 + c.p] = 0.0;
    tr.fy2[c.q0 + c.p] = 0.0;
  } else if (!edge_face(c.j, a.es, a.en)) {
    const double* line = tr.qc2 + c.q0;
    auto xv = [&](int m) { return line[pg.at(c.i, m)]; };
    tr.fy2[c.q0 + c.p] =
        face_weights(a.hord, a.lim_fac, c.j, xv, a.cy[c.lev + c.p], tr.wyi + c.q0 + c.p, ws, a.odd);
  }
  if (!xi_face(a, c.i, c.j)) {
    for (int s = 0; s < 6; ++s) tr.wxi[s * ws + c.q0 + c.p] = 0.0;
    tr.fx2[c.q0 + c.p] = 0.0;
  } else if (!edge_face(c.i, a.ew, a.ee)) {
    const double* line = tr.qc1 + c.q0;
    auto xv = [&](int m) { return line[pg.at(m, c.j)]; };
    tr.fx2[c.q0 + c.p] =
        face_weights(a.hord, a.lim_fac, c.i, xv, a.cx[c.lev + c.p], tr.wxi + c.q0 + c.p, ws, a.odd);
  }
}

// Faces beside the cube-face edges of both sweeps of a pass (inner: x on the
// dir-1 copy, y on the dir-2 copy; outer: x on q_i, y on q_j), a thread per
// line, edge and face around it (10 faces of a line): compact, so that the
// few one-sided faces do not hold up warps of ordinary ones.  blockIdx.z: 0 x
// faces, 1 y faces.
__global__ void k_lin_edges(const LinArgs a, const LinTraj tr, int outer) {
  const bool ydir = blockIdx.z == 1;
  const int lo = ydir ? (outer ? a.is : a.isd) : (outer ? a.js : a.jsd);
  const int hi = ydir ? (outer ? a.ie : a.ied) : (outer ? a.je : a.jed);
  const int nlines = hi - lo + 1;
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= nlines * 10) return;
  const int line = lo + id % nlines, slot = id / nlines;
  const int eLo = ydir ? a.es : a.ew, eHi = ydir ? a.en : a.ee;
  const int e = slot < 5 ? eLo : eHi;
  if (e == NO_EDGE) return;
  const int f = e - 2 + slot % 5;
  if (!in_rng(f, ydir ? a.js : a.is, (ydir ? a.je : a.ie) + 1)) return;
  const PlaneGeom& pg = a.pg;
  const long long ws = (long long)a.nt * a.nq * a.npz * a.P;
  const int pl = blockIdx.y, per_tile = a.nq * a.npz;
  const int t = pl / per_tile;
  const long long q0 = (long long)pl * a.P, lev = ((long long)t * a.npz + pl % a.npz) * a.P, met = (long long)t * a.P;
  const long long p = ydir ? pg.at(line, f) : pg.at(f, line);
  const double* src = (outer ? (ydir ? tr.qj : tr.qi) : (ydir ? tr.qc2 : tr.qc1)) + q0;
  const double* da = (ydir ? a.dya : a.dxa) + met;
  double* w = (outer ? (ydir ? tr.wyo : tr.wxo) : (ydir ? tr.wyi : tr.wxi)) + q0 + p;
  auto at = [&](int m) { return ydir ? pg.at(line, m) : pg.at(m, line); };
  auto xv = [&](int m) { return src[at(m)]; };
  auto dx = [&](int m) { return da[at(m)]; };
  const double fl = edge_face_weights(a.hord, a.lim_fac, f, xv, dx, (ydir ? a.cy : a.cx)[lev + p], eLo, eHi, w, ws,
                                      a.odd);
  if (!outer) (ydir ? tr.fy2 : tr.fx2)[q0 + p] = fl;
}

// Faces with an infinity or a NaN in their window or Courant number: the same by forward-mode
// passes, after the kernels of a pass reported one in a.odd (else this ends at once: 12
// launches in a step of six substeps).
__global__ void __launch_bounds__(128) k_lin_odd(const LinArgs a, const LinTraj tr, int outer) {
  if (*a.odd == 0) return;
  const PlaneGeom& pg = a.pg;
  const long long ws = (long long)a.nt * a.nq * a.npz * a.P, n = 2 * ws;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const bool ydir = e >= ws;
    const long long id = ydir ? e - ws : e, p = id % a.P, pl = id / a.P, q0 = pl * a.P;
    const int per_tile = a.nq * a.npz, t = (int)(pl / per_tile);
    const long long lev = ((long long)t * a.npz + pl % a.npz) * a.P, met = (long long)t * a.P;
    const int i = pg.isd + (int)(p % pg.pitch), j = pg.jsd + (int)(p / pg.pitch);
    if (!(ydir ? (outer ? yo_face(a, i, j) : yi_face(a, i, j)) : (outer ? xo_face(a, i, j) : xi_face(a, i, j)))) continue;
    const double* src = (outer ? (ydir ? tr.qj : tr.qi) : (ydir ? tr.qc2 : tr.qc1)) + q0;
    const double* da = (ydir ? a.dya : a.dxa) + met;
    const double c = (ydir ? a.cy : a.cx)[lev + p];
    const int f = ydir ? j : i;
    auto xv = [&](int m) { return src[ydir ? pg.at(i, m) : pg.at(m, j)]; };
    auto dx = [&](int m) { return da[ydir ? pg.at(i, m) : pg.at(m, j)]; };
    double x[6];
    for (int s = 0; s < 6; ++s) x[s] = xv(f - 3 + s);
    if (!odd_window(x, c)) continue;
    double* w = (outer ? (ydir ? tr.wyo : tr.wxo) : (ydir ? tr.wyi : tr.wxi)) + q0 + p;
    const double fl = forward_weights(a.hord, a.lim_fac, f, xv, dx, c, ydir ? a.es : a.ew, ydir ? a.en : a.ee, w, ws);
    if (!outer) (ydir ? tr.fy2 : tr.fx2)[q0 + p] = fl;
  }
}

// Inner updates: q_i = (q area + yfx fy2 - yfx' fy2') / ra_y on the compute
// rows of every column, q_j likewise along x on the compute columns of every
// row.  The same form maps the tangents.
__global__ void k_lin_mid(const LinArgs a, const double* c1, const double* c2, const double* fx2, const double* fy2,
                          double* qi, double* qj) {
  Cell c;
  if (!cell_of(a, c)) return;
  const int i = c.i, j = c.j;
  const PlaneGeom& pg = a.pg;
  double vi = 0.0, vj = 0.0;
  if (in_rng(j, a.js, a.je)) {
    const double y0 = a.yfx[c.lev + pg.at(i, j)], y1 = a.yfx[c.lev + pg.at(i, j + 1)];
    vi = (c2[c.q0 + c.p] * a.area[c.met + c.p] + y0 * fy2[c.q0 + pg.at(i, j)] - y1 * fy2[c.q0 + pg.at(i, j + 1)]) *
         inv_ra_y(a, c, i, j);
  }
  if (in_rng(i, a.is, a.ie)) {
    const double x0 = a.xfx[c.lev + pg.at(i, j)], x1 = a.xfx[c.lev + pg.at(i + 1, j)];
    vj = (c1[c.q0 + c.p] * a.area[c.met + c.p] + x0 * fx2[c.q0 + pg.at(i, j)] - x1 * fx2[c.q0 + pg.at(i + 1, j)]) *
         inv_ra_x(a, c, i, j);
  }
  qi[c.q0 + c.p] = vi;
  qj[c.q0 + c.p] = vj;
}

// Outer sweeps: x faces of the compute rows on q_i, y faces of the compute
// columns on q_j: weights (faces beside a cube-face edge: k_lin_edges).
__global__ void k_lin_outer(const LinArgs a, const LinTraj tr) {
  Cell c;
  if (!cell_of(a, c)) return;
  const long long ws = (long long)a.nt * a.nq * a.npz * a.P;
  const PlaneGeom& pg = a.pg;
  if (!xo_face(a, c.i, c.j)) {
    for (int s = 0; s < 6; ++s) tr.wxo[s * ws + c.q0 + c.p] = 0.0;
  } else if (!edge_face(c.i, a.ew, a.ee)) {
    const double* line = tr.qi + c.q0;
    auto xv = [&](int m) { return line[pg.at(m, c.j)]; };
    face_weights(a.hord, a.lim_fac, c.i, xv, a.cx[c.lev + c.p], tr.wxo + c.q0 + c.p, ws, a.odd);
  }
  if (!yo_face(a, c.i, c.j)) {
    for (int s = 0; s < 6; ++s) tr.wyo[s * ws + c.q0 + c.p] = 0.0;
  } else if (!edge_face(c.j, a.es, a.en)) {
    const double* line = tr.qj + c.q0;
    auto xv = [&](int m) { return line[pg.at(c.i, m)]; };
    face_weights(a.hord, a.lim_fac, c.j, xv, a.cy[c.lev + c.p], tr.wyo + c.q0 + c.p, ws, a.odd);
  }
}

// ------------------------------------------------------- tangent-linear ---
// Inner-sweep flux tangents from the corner-filled tangents.
__global__ void k_tl_inner(const LinArgs a, const LinTraj tr, const double* t1, const double* t2, double* fx2,
                           double* fy2) {
  Cell c;
  if (!cell_of(a, c)) return;
  const long long ws = (long long)a.nt * a.nq * a.npz * a.P;
  const PlaneGeom& pg = a.pg;
  double fy = 0.0, fx = 0.0;
  if (yi_face(a, c.i, c.j))
    for (int s = 0; s < 6; ++s) fy += tr.wyi[s * ws + c.q0 + c.p] * t2[c.q0 + pg.at(c.i, c.j - 3 + s)];
  if (xi_face(a, c.i, c.j))
    for (int s = 0; s < 6; ++s) fx += tr.wxi[s * ws + c.q0 + c.p] * t1[c.q0 + pg.at(c.i - 3 + s, c.j)];
  fy2[c.q0 + c.p] = fy;
  fx2[c.q0 + c.p] = fx;
}

// The substep's update of a compute cell from the outer-sweep flux tangents
// (computed here for the cell's four faces) and the inner ones.
__global__ void k_tl_update(const LinArgs a, const LinTraj tr, const double* dq, const double* ti, const double* tj,
                            const double* fx2, const double* fy2, double* out) {
  Cell c;
  if (!cell_of(a, c)) return;
  const long long ws = (long long)a.nt * a.nq * a.npz * a.P;
  const int i = c.i, j = c.j;
  const PlaneGeom& pg = a.pg;
  if (!in_rng(i, a.is, a.ie) || !in_rng(j, a.js, a.je)) {
    out[c.q0 + c.p] = 0.0;
    return;
  }
  auto FX = [&](int f) {
    const long long pf = pg.at(f, j);
    double fo = 0.0;
    for (int s = 0; s < 6; ++s) fo += tr.wxo[s * ws + c.q0 + pf] * ti[c.q0 + pg.at(f - 3 + s, j)];
    return (fo + fx2[c.q0 + pf]) * (0.5 * a.mfx[c.lev + pf]);
  };
  auto FY = [&](int f) {
    const long long pf = pg.at(i, f);
    double fo = 0.0;
    for (int s = 0; s < 6; ++s) fo += tr.wyo[s * ws + c.q0 + pf] * tj[c.q0 + pg.at(i, f - 3 + s)];
    return (fo + fy2[c.q0 + pf]) * (0.5 * a.mfy[c.lev + pf]);
  };
  const double div = FX(i) - FX(i + 1) + FY(j) - FY(j + 1);
  out[c.q0 + c.p] = fma(dq[c.q0 + c.p], a.dr[c.lev + c.p], div * a.r2[c.lev + c.p]);
}

// ------------------------------------------------------------- adjoint ---
// Outer-sweep flux adjoints of the substep: with t = q_ad rarea / dp2 on the
// compute cells, FX_ad(f) = t(f) - t(f-1), and both x sweeps' fluxes enter
// FX with 0.5 mfx.
__global__ void k_ad_faces(const LinArgs a, const double* qa, double* gx, double* gy) {
  Cell c;
  if (!cell_of(a, c)) return;
  const int i = c.i, j = c.j;
  const PlaneGeom& pg = a.pg;
  auto tt = [&](int ii, int jj) -> double {
    if (!in_rng(ii, a.is, a.ie) || !in_rng(jj, a.js, a.je)) return 0.0;
    const long long p = pg.at(ii, jj);
    return qa[c.q0 + p] * a.r2[c.lev + p];
  };
  double vx = 0.0, vy = 0.0;
  if (xo_face(a, i, j)) vx = 0.5 * a.mfx[c.lev + c.p] * (tt(i, j) - tt(i - 1, j));
  if (yo_face(a, i, j)) vy = 0.5 * a.mfy[c.lev + c.p] * (tt(i, j) - tt(i, j - 1));
  gx[c.q0 + c.p] = vx;
  gy[c.q0 + c.p] = vy;
}

// The same from fv_tp_2d's flux adjoints: g = 0.5 w flux_ad.
__global__ void k_ad_flux_in(const LinArgs a, const double* fxa, const double* fya, double* gx, double* gy) {
  Cell c;
  if (!cell_of(a, c)) return;
  gx[c.q0 + c.p] = xo_face(a, c.i, c.j) ? 0.5 * a.mfx[c.lev + c.p] * fxa[c.q0 + c.p] : 0.0;
  gy[c.q0 + c.p] = yo_face(a, c.i, c.j) ? 0.5 * a.mfy[c.lev + c.p] * fya[c.q0 + c.p] : 0.0;
}

// Outer sweeps transposed: the adjoints of q_i (compute rows, every column)
// and of q_j (compute columns, every row), each cell summing the faces whose
// stencils hold it.
__global__ void k_ad_outer(const LinArgs a, const LinTraj tr, const double* gx, const double* gy, double* ai,
                           double* aj) {
  Cell c;
  if (!cell_of(a, c)) return;
  const long long ws = (long long)a.nt * a.nq * a.npz * a.P;
  const int i = c.i, j = c.j;
  const PlaneGeom& pg = a.pg;
  double vi = 0.0, vj = 0.0;
  if (in_rng(j, a.js, a.je))
    for (int f = max(a.is, i - 2); f <= min(a.ie + 1, i + 3); ++f) {
      const long long pf = pg.at(f, j);
      vi += tr.wxo[(i - f + 3) * ws + c.q0 + pf] * gx[c.q0 + pf];
    }
  if (in_rng(i, a.is, a.ie))
    for (int f = max(a.js, j - 2); f <= min(a.je + 1, j + 3); ++f) {
      const long long pf = pg.at(i, f);
      vj += tr.wyo[(j - f + 3) * ws + c.q0 + pf] * gy[c.q0 + pf];
    }
  ai[c.q0 + c.p] = vi;
  aj[c.q0 + c.p] = vj;
}

// Inner updates transposed, flux part: the adjoints of the inner-sweep
// fluxes (their direct share of FX, FY plus their terms in q_i, q_j).
__global__ void k_ad_mid(const LinArgs a, const double* ai, const double* aj, const double* gx, const double* gy,
                         double* fx2, double* fy2) {
  Cell c;
  if (!cell_of(a, c)) return;
  const int i = c.i, j = c.j;
  const PlaneGeom& pg = a.pg;
  double vy = 0.0, vx = 0.0;
  if (yi_face(a, i, j)) {
    double s = 0.0;
    if (j <= a.je) s += ai[c.q0 + pg.at(i, j)] * inv_ra_y(a, c, i, j);
    if (j - 1 >= a.js) s -= ai[c.q0 + pg.at(i, j - 1)] * inv_ra_y(a, c, i, j - 1);
    vy = a.yfx[c.lev + c.p] * s + (in_rng(i, a.is, a.ie) ? gy[c.q0 + c.p] : 0.0);
  }
  if (xi_face(a, i, j)) {
    double s = 0.0;
    if (i <= a.ie) s += aj[c.q0 + pg.at(i, j)] * inv_ra_x(a, c, i, j);
    if (i - 1 >= a.is) s -= aj[c.q0 + pg.at(i - 1, j)] * inv_ra_x(a, c, i - 1, j);
    vx = a.xfx[c.lev + c.p] * s + (in_rng(j, a.js, a.je) ? gx[c.q0 + c.p] : 0.0);
  }
  fy2[c.q0 + c.p] = vy;
  fx2[c.q0 + c.p] = vx;
}

// Inner sweeps transposed: the adjoints of the two corner-filled copies
// (their area terms in q_i, q_j plus the gathered stencil terms).
__global__ void k_ad_inner(const LinArgs a, const LinTraj tr, const double* ai, const double* aj, const double* fx2,
                           const double* fy2, double* a1, double* a2) {
  Cell c;
  if (!cell_of(a, c)) return;
  const long long ws = (long long)a.nt * a.nq * a.npz * a.P;
  const int i = c.i, j = c.j;
  const PlaneGeom& pg = a.pg;
  double v1 = 0.0, v2 = 0.0;
  if (in_rng(j, a.js, a.je)) v2 = ai[c.q0 + c.p] * a.area[c.met + c.p] * inv_ra_y(a, c, i, j);
  for (int f = max(a.js, j - 2); f <= min(a.je + 1, j + 3); ++f) {
    const long long pf = pg.at(i, f);
    v2 += tr.wyi[(j - f + 3) * ws + c.q0 + pf] * fy2[c.q0 + pf];
  }
  if (in_rng(i, a.is, a.ie)) v1 = aj[c.q0 + c.p] * a.area[c.met + c.p] * inv_ra_x(a, c, i, j);
  for (int f = max(a.is, i - 2); f <= min(a.ie + 1, i + 3); ++f) {
    const long long pf = pg.at(f, j);
    v1 += tr.wxi[(i - f + 3) * ws + c.q0 + pf] * fx2[c.q0 + pf];
  }
  a1[c.q0 + c.p] = v1;
  a2[c.q0 + c.p] = v2;
}

// The input's adjoint before the corner (and halo) transposes: the substep's
// direct term dp1/dp2 on the compute cells (qa, when given) plus both
// copies' adjoints off the filled corner blocks; added to out when acc.
__global__ void k_ad_collect(const LinArgs a, const double* qa, const double* a1, const double* a2, double* out,
                             int acc) {
  Cell c;
  if (!cell_of(a, c)) return;
  double v = 0.0;
  if (qa && in_rng(c.i, a.is, a.ie) && in_rng(c.j, a.js, a.je))
    v = qa[c.q0 + c.p] * a.dr[c.lev + c.p];
  if (!corner_cell(a, c.i, c.j)) v += a1[c.q0 + c.p] + a2[c.q0 + c.p];
  out[c.q0 + c.p] = acc ? out[c.q0 + c.p] + v : v;
}

// copy_corners transposed: each filled corner-block cell's adjoint moves to
// the halo-strip cell it was rotated from (one thread per plane and corner;
// the 72 rotation targets of a plane are distinct, so no two threads meet).
__global__ void k_ad_corners(const LinArgs a, const double* a1, const double* a2, double* out) {
  const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nplanes = (long long)a.nt * a.nq * a.npz;
  if (id >= nplanes * 4) return;
  const long long q0 = (id / 4) * a.P;
  const int corner = (int)(id % 4);
  if (!((a.corners >> corner) & 1)) return;
  const int ib = (corner & 1) ? a.npx : 1 - NG, jb = (corner & 2) ? a.npy : 1 - NG;
  for (int dj = 0; dj < NG; ++dj)
    for (int di = 0; di < NG; ++di) {
      const int i = ib + di, j = jb + dj;
      if (!inside_data(a, i, j)) continue;
      const long long p = a.pg.at(i, j);
      int i1 = i, j1 = j, i2 = i, j2 = j;
      corner_rotate(i1, j1, a.npx, a.npy, 1);
      corner_rotate(i2, j2, a.npx, a.npy, 2);
      if (inside_data(a, i1, j1)) out[q0 + a.pg.at(i1, j1)] += a1[q0 + p];
      if (inside_data(a, i2, j2)) out[q0 + a.pg.at(i2, j2)] += a2[q0 + p];
    }
}

// Cube halo transposed: every interior cell within NG of a tile edge adds the
// adjoints of the halo cells of the neighbouring tiles that copy it; halo
// cells leave with zero.
__global__ void k_ad_halo(const LinArgs a, const double* in, double* out) {
  Cell c;
  if (!cell_of(a, c)) return;
  const int n = a.n, i = c.i, j = c.j;
  if (i < 1 || i > n || j < 1 || j > n) {
    out[c.q0 + c.p] = 0.0;
    return;
  }
  double v = in[c.q0 + c.p];
  const long long per_tile = (long long)a.nq * a.npz;
  const long long within = c.pl - (long long)c.t * per_tile;  // tracer and level inside the tile
  for (int e = 0; e < 4; ++e) {
    int d, sb;
    switch (e) {
      case EW: d = i; sb = j - 1; break;
      case EE: d = n + 1 - i; sb = j - 1; break;
      case ES: d = j; sb = i - 1; break;
      default: d = n + 1 - j; sb = i - 1; break;
    }
    if (d > NG) continue;
    const int u = a.topo.nbr[c.t][e], fe = a.topo.nedge[c.t][e];
    const int su = a.topo.rev[u][fe] ? n - 1 - sb : sb;
    int hi, hj;
    switch (fe) {
      case EW: hi = 1 - d; hj = su + 1; break;
      case EE: hi = n + d; hj = su + 1; break;
      case ES: hi = su + 1; hj = 1 - d; break;
      default: hi = su + 1; hj = n + d; break;
    }
    v += in[((long long)u * per_tile + within) * a.P + a.pg.at(hi, hj)];
  }
  out[c.q0 + c.p] = v;
}

// del-2 damping fluxes transposed (fluxes d6 (q(m-1) - q(m)) through the
// compute faces): q_ad(m) += d6(m+1) F_ad(m+1) - d6(m) F_ad(m) along x and y.
__global__ void k_ad_damp(const LinArgs a, const double* fxa, const double* fya, const double* d6x,
                          const double* d6y, double* out) {
  Cell c;
  if (!cell_of(a, c)) return;
  const int i = c.i, j = c.j;
  const PlaneGeom& pg = a.pg;
  double v = 0.0;
  if (d6x && in_rng(j, a.js, a.je)) {
    if (xo_face(a, i + 1, j)) v += d6x[pg.at(i + 1, j)] * fxa[c.q0 + pg.at(i + 1, j)];
    if (xo_face(a, i, j)) v -= d6x[pg.at(i, j)] * fxa[c.q0 + pg.at(i, j)];
  }
  if (d6y && in_rng(i, a.is, a.ie)) {
    if (yo_face(a, i, j + 1)) v += d6y[pg.at(i, j + 1)] * fya[c.q0 + pg.at(i, j + 1)];
    if (yo_face(a, i, j)) v -= d6y[pg.at(i, j)] * fya[c.q0 + pg.at(i, j)];
  }
  out[c.q0 + c.p] += v;
}

dim3 plane_grid(const LinArgs& a) {
  return dim3((unsigned)((a.P + 127) / 128), (unsigned)(a.nt * a.nq * a.npz));
}

// ------------------------------------------------ remap reverse (kord 4) ---
// One column's source means, slopes, interfaces, the overlap schedule and
// the adjoints, in local memory.
struct ColumnAd {
  static constexpr bool DUAL = false;
  double q[KMAX], h[KMAX], d[KMAX], a[KMAX + 1];
  double qa[KMAX], da[KMAX], aa[KMAX + 1];
  double pl[KMAX], pr[KMAX], p6[KMAX];  // adjoints of the layer parabolas (left, right edge, curvature)
  double x[KMAX + 1];
  unsigned char L[KMAX + 1];
};

// d pmean(l, r, s6, x1, x2) / d(l, r, s6), pmean the mean of the layer's
// parabola over the fraction [x1, x2]
__device__ __forceinline__ void pmean_grad(double x1, double x2, double g, double& gl, double& gr, double& g6) {
  const double m = 0.5 * (x1 + x2);
  gl += g * (1.0 - m);
  gr += g * m;
  g6 += g * (m - (x2 * x2 + x1 * x2 + x1 * x1) * (1.0 / 3.0));
}

constexpr double kNaN = __builtin_nan("");

// ---- local derivatives of the kord-4 scheme (fv3g_profile.cuh) at the trajectory,
// every branch frozen; on a tie the later operand, as min, max and the tests on
// dual numbers take it.  The columns are bound by FP64 instructions and their per-thread
// arrays: a forward-mode pass per input of every layer, interface and slope took 28.8 ms
// for six C96 tiles x 64 levels x 4 tracers, these 6.5 ms (reverse) and, instead of the
// column kernel on dual numbers, 6.2 ms (tangent; 12.0 ms).

// slope4_grad with an infinity or a NaN among the means, in forward mode.
template <bool DUAL>
__device__ __noinline__ double slope4_odd(double qm, double q0, double qp, double d0, double d1, double d2, double* p) {
  D2 r;
  for (int s = 0; s < 3; ++s) {
    r = ppm_slope(D2(qm, s == 0 ? 1.0 : 0.0), D2(q0, s == 1 ? 1.0 : 0.0), D2(qp, s == 2 ? 1.0 : 0.0), D2(d0), D2(d1), D2(d2));
    p[s] = r.d;
  }
  return DUAL ? r.v : ppm_slope<double>(qm, q0, qp, d0, d1, d2);
}
// d slope / d (qm, q0, qp) and the slope of a layer from the means and thicknesses of
// the layer and its neighbours.  DUAL: beside an infinity or a NaN the value is that of the dual
// numbers (the tangent's columns), whose comparisons choose otherwise than fmin and fmax.
// ODD, here and below: the column may hold infinities or NaN (a kernel of its own for those).
template <bool ODD, bool DUAL = false>
__device__ __forceinline__ double slope4_grad(double qm, double q0, double qp, double d0, double d1, double d2,
                                              double* p) {
  if (ODD && (inf_or_nan(qm) || inf_or_nan(q0) || inf_or_nan(qp))) return slope4_odd<DUAL>(qm, q0, qp, d0, d1, d2, p);
  const double f = d1 * fast_rcp(d0 + d1 + d2);
  const double A = f * ((2.0 * d0 + d1) * fast_rcp(d2 + d1)), B = f * ((d1 + 2.0 * d2) * fast_rcp(d0 + d1));
  const double Dm = q0 - qm, Dp = qp - q0, s = qp - qm;
  const double dq = fma(A, Dp, B * Dm), half = scale2<-1>(absv(dq));
  const bool hi_m = neg(Dm) && neg(s), hi_0 = !neg(Dm) && neg(Dp);
  const bool lo_m = pos(Dm) && pos(s), lo_0 = !pos(Dm) && pos(Dp);
  const double mx = hi_m ? negv(Dm) : hi_0 ? 0.0 : Dp, mn = lo_m ? Dm : lo_0 ? 0.0 : absv(Dp);
  const bool use_h = mag_less(half, mx);
  const double m1 = use_h ? half : mx;
  const bool use_1 = mag_less(m1, mn);
  const bool ng = neg(dq);
  const double sg = ng ? -1.0 : 1.0, hA = 0.5 * A, hB = 0.5 * B;
  if (!use_1) {
    p[0] = lo_m ? -sg : 0.0;
    p[1] = lo_0 ? 0.0 : sg;
    p[2] = (lo_m || lo_0) ? 0.0 : -sg;
  } else if (use_h) {
    p[0] = negv(hB);
    p[1] = hB - hA;
    p[2] = hA;
  } else {
    p[0] = hi_m ? sg : 0.0;
    p[1] = hi_0 ? 0.0 : -sg;
    p[2] = (hi_m || hi_0) ? 0.0 : sg;
  }
  const double m = absv(use_1 ? m1 : mn);
  return ng ? negv(m) : m;
}

// Interface u as a linear form: means of layers lo, lo+1, lo+2 and (inside) the
// slopes dl, dr of layers u-1, u.
struct InterfaceDer {
  double q[3], dl, dr;
  int lo;
  bool inner;
};
__device__ __forceinline__ bool inner_interface(int u, int km) { return km > 2 && u >= 2 && u <= km - 2; }
// an infinity or a NaN in what interface u reads (dml, dmr: the slopes of layers u-1, u)
template <class QF>
__device__ __forceinline__ bool odd_interface(int u, int km, const QF& q, double dml, double dmr) {
  if (inner_interface(u, km)) return inf_or_nan(q(u - 1)) || inf_or_nan(q(u)) || inf_or_nan(dml) || inf_or_nan(dmr);
  const int lo = u <= 1 ? 0 : km - 3;
  return inf_or_nan(q(lo)) || inf_or_nan(q(lo + 1)) || inf_or_nan(q(lo + 2));
}
// its derivatives in forward mode
template <class QF, class HF>
__device__ __noinline__ InterfaceDer interface_odd(int u, int km, int iv, QF q, HF h, double dml, double dmr) {
  InterfaceDer D{{0.0, 0.0, 0.0}, 0.0, 0.0, 0, inner_interface(u, km)};
  D.lo = D.inner ? u - 1 : u <= 1 || km == 2 ? 0 : km - 3;
  enum { SLOPE_L = 1000, SLOPE_R };  // seeds beside the means' 0..2
  auto pass = [&](int s) -> double {
    auto qd = [&](int k) -> D2 { return D2(q(k), min(max(k, 0), km - 1) == D.lo + s ? 1.0 : 0.0); };
    auto hd = [&](int k) -> D2 { return D2(h(k)); };
    return ppm_interface<D2>(u, km, iv, D2(0.0), D2(dml, s == SLOPE_L ? 1.0 : 0.0), D2(dmr, s == SLOPE_R ? 1.0 : 0.0), qd, hd).d;
  };
  for (int s = 0; s < (D.inner || km == 2 ? 2 : 3); ++s) D.q[s] = pass(s);
  if (D.inner) {
    D.dl = pass(SLOPE_L);
    D.dr = pass(SLOPE_R);
  }
  return D;
}
template <bool ODD, class QF, class HF>
__device__ InterfaceDer interface_der(int u, int km, int iv, const QF& q, const HF& h, double dml, double dmr) {
  if (ODD && odd_interface(u, km, q, dml, dmr)) return interface_odd(u, km, iv, q, h, dml, dmr);
  InterfaceDer D{{0.0, 0.0, 0.0}, 0.0, 0.0, 0, false};
  if (inner_interface(u, km)) {
    const double hm = h(u - 2), h0 = h(u - 1), h1 = h(u), h2 = h(u + 1);
    const double pair = fast_rcp(h0 + h1), sall = fast_rcp(hm + h0 + h1 + h2);
    const double fa = (hm + h0) * fast_rcp(2.0 * h0 + h1), fb = (h2 + h1) * fast_rcp(2.0 * h1 + h0);
    const double c = h0 * pair + 2.0 * h1 * h0 * pair * (fa - fb) * sall;
    D.q[0] = 1.0 - c;
    D.q[1] = c;
    D.dr = -2.0 * h0 * fa * sall;
    D.dl = 2.0 * h1 * fb * sall;
    D.lo = u - 1;
    D.inner = true;
    return D;
  }
  if (u >= km && iv == -2) return D;  // the given surface value
  if (km == 2) {
    const double w0 = h(1) / (h(0) + h(1)), w1 = h(0) / (h(0) + h(1));
    D.q[0] = u == 1 ? w0 : u <= 0 ? 2.0 - w0 : -w0;
    D.q[1] = u == 1 ? w1 : u <= 0 ? -w1 : 2.0 - w1;
    return D;
  }
  // the parabola through the three layers at the end, clamped into the two beside the interface
  const bool top = u <= 1;
  const int k0 = top ? 0 : km - 1, k1 = top ? 1 : km - 2, k2 = top ? 2 : km - 3;
  const double h0 = h(k0), h1 = h(k1), h2 = h(k2), x0 = top ? q(k0) : q(k1), x1 = top ? q(k1) : q(k0);
  const double w0 = h1 * (h1 + h2) / ((h0 + h1) * (h0 + h1 + h2)), w2 = -h0 * h1 / ((h0 + h1 + h2) * (h1 + h2));
  const double w1 = 1.0 - w0 - w2, v = w0 * q(k0) + w1 * q(k1) + w2 * q(k2);
  const double lo = x0 < x1 ? x0 : x1, hi = x0 > x1 ? x0 : x1, vl = v > lo ? v : lo;
  double e0 = 0.0, e1 = 0.0, e2 = 0.0;  // on k0, k1, k2
  if (vl < hi) {
    if (v > lo) {
      e0 = w0;
      e1 = w1;
      e2 = w2;
    } else if ((x0 < x1) == top) {
      e0 = 1.0;
    } else {
      e1 = 1.0;
    }
  } else if ((x0 > x1) == top) {
    e0 = 1.0;
  } else {
    e1 = 1.0;
  }
  if (u <= 0 || u >= km) {  // the outermost interface: 2 q less the next one
    e0 = 2.0 - e0;
    e1 = -e1;
    e2 = -e2;
  }
  D.lo = top ? 0 : km - 3;
  D.q[0] = top ? e0 : e2;
  D.q[1] = e1;
  D.q[2] = top ? e2 : e0;
  return D;
}

// d bl, d br of a layer's limited edge deviations: l[0] (d aL - d q) + l[1] (d aR - d
// q) + l[2] d slope, r likewise; low: the positivity scaling acts, or an infinity or a NaN
// comes in (layer_der_low).
struct LayerDer {
  double l[3], r[3];
  bool low;
};
template <bool ODD>
__device__ __forceinline__ LayerDer layer_der(bool inner, double q, double aL, double aR, double d, int iv,
                                              double floor_v) {
  LayerDer D{{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}, false};
  if (ODD && (inf_or_nan(q) || inf_or_nan(aL) || inf_or_nan(aR) || inf_or_nan(d))) {
    D.low = true;
    return D;
  }
  const double b0 = aL - q, r0 = aR - q;
  double bl, br;
  if (inner) {  // Lin (2004): at most |2 d| with the sign of d
    const double ax = scale2<1>(absv(d));
    const bool nd = neg(d), lim_l = mag_less(ax, absv(b0)), lim_r = mag_less(ax, absv(r0));
    const double ml = lim_l ? ax : absv(b0), mr = lim_r ? ax : absv(r0);
    bl = nd ? ml : negv(ml);
    br = nd ? negv(mr) : mr;
    if (lim_l) D.l[2] = -2.0;
    else D.l[0] = nd == neg(b0) ? -1.0 : 1.0;
    if (lim_r) D.r[2] = 2.0;
    else D.r[1] = nd == neg(r0) ? 1.0 : -1.0;
  } else {  // CW84 eq. 1.10
    bl = b0;
    br = r0;
    const bool flat = !opposite(b0, r0);
    const double dd = r0 - b0, t = 3.0 * dd * (b0 + r0), d2 = dd * dd;
    const bool lo = -t > d2, hi = !lo && t > d2;
    if (flat) {
      bl = br = 0.0;
    } else if (lo) {
      bl = -2.0 * r0;
      D.l[1] = -2.0;
      D.r[1] = 1.0;
    } else if (hi) {
      br = -2.0 * b0;
      D.l[0] = 1.0;
      D.r[0] = -2.0;
    } else {
      D.l[0] = 1.0;
      D.r[1] = 1.0;
    }
  }
  if (iv >= 0) {
    // below the floor at an edge, or inside where bl + br exceeds the mean's height above the floor
    const double s = bl + br, qf = floor_v == 0.0 ? q : q - floor_v;
    D.low = less(q + bl, floor_v) || less(q + br, floor_v) || (pos(s) && less(qf, s));
  }
  return D;
}
// The layer's (l, r, s6) by (q, aL, aR, d) in forward mode: layers near the floor, or beside a NaN.
// Returns whether the parabola's values (as its mean takes them) are finite.
__device__ __noinline__ bool layer_der_low(int k, int km, double q, double aL, double aR, double d, int iv,
                                           double floor_v, double (*J)[4]) {
  bool finite = true;
  for (int s = 0; s < 4; ++s) {
    const D2 qd(q, s == 0 ? 1.0 : 0.0);
    const Profile<D2> P = layer_profile<D2, 4>(k, km, qd, qd, qd, qd, qd, D2(aL, s == 1 ? 1.0 : 0.0),
                                               D2(aR, s == 2 ? 1.0 : 0.0), D2(d, s == 3 ? 1.0 : 0.0), iv, D2(floor_v));
    J[0][s] = P.l.d;
    J[1][s] = P.r.d;
    J[2][s] = P.s6.d;
    finite = !inf_or_nan(P.s6.v) && !inf_or_nan((P.r.v - P.l.v) + P.s6.v);
  }
  return finite;
}

// Slopes C.d and interface values C.a of the trajectory (C.q, C.h).
template <bool ODD, class CC, class QF, class HF>
__device__ void column_forward4(CC& C, int km, int iv, double qs, const QF& qf, const HF& hf) {
  double p[3];
  for (int k = 0; k < km; ++k)
    C.d[k] = k < 1 || k > km - 2
                 ? 0.0
                 : slope4_grad<ODD, CC::DUAL>(C.q[k - 1], C.q[k], C.q[k + 1], C.h[k - 1], C.h[k], C.h[k + 1], p);
  for (int u = 0; u <= km; ++u) {
    const double dml = u >= 1 ? C.d[u - 1] : 0.0, dmr = u < km ? C.d[u] : 0.0;
    if (inner_interface(u, km) && !(ODD && odd_interface(u, km, qf, dml, dmr))) {
      const InterfaceDer D = interface_der<false>(u, km, iv, qf, hf, dml, dmr);
      C.a[u] = fma(D.q[1], C.q[u] - C.q[u - 1], C.q[u - 1]) + fma(D.dr, C.d[u], D.dl * C.d[u - 1]);
    } else if (ODD && CC::DUAL) {
      auto qd = [&](int k) -> D2 { return D2(qf(k)); };
      auto hd = [&](int k) -> D2 { return D2(hf(k)); };
      C.a[u] = ppm_interface<D2>(u, km, iv, D2(qs), D2(dml), D2(dmr), qd, hd).v;
    } else {
      C.a[u] = ppm_interface<double>(u, km, iv, qs, dml, dmr, qf, hf);
    }
  }
}

__device__ __forceinline__ bool odd_column(const double* q, int km) {
  bool odd = false;
  for (int k = 0; k < km; ++k) odd |= inf_or_nan(q[k]);
  return odd;
}

// Reverse of one column: pe1(k) (k = 0..km) source interface pressures,
// pe2(k) target ones, G2(k2) the target adjoints; leaves the source
// adjoints in C.qa.  C.q holds the source means.
template <bool ODD, class PE1, class PE2, class G2>
__device__ void column_ad4(ColumnAd& C, int km, int kn, int iv, double floor_v, double qs, const PE1& pe1,
                           const PE2& pe2, const G2& g2) {
  // thicknesses and the overlap schedule, as the forward kernel forms them
  {
    double p1 = pe1(0);
    for (int k = 0; k < km; ++k) {
      const double p2 = pe1(k + 1);
      C.h[k] = p2 - p1;
      p1 = p2;
    }
    int k1 = 0;
    double lo = pe1(0), hi = pe1(1);
    for (int k2 = 0; k2 <= kn; ++k2) {
      const double p = pe2(k2);
      while (k1 < km - 1 && hi <= p) {
        ++k1;
        lo = hi;
        hi = pe1(k1 + 1);
      }
      C.L[k2] = (unsigned char)k1;
      C.x[k2] = fast_div(p - lo, hi - lo);
    }
  }
  auto qf = [&](int k) -> double { return C.q[min(max(k, 0), km - 1)]; };
  auto hf = [&](int k) -> double { return C.h[min(max(k, 0), km - 1)]; };
  column_forward4<ODD>(C, km, iv, qs, qf, hf);
  for (int k = 0; k < km; ++k) C.qa[k] = C.da[k] = C.pl[k] = C.pr[k] = C.p6[k] = 0.0;
  for (int u = 0; u <= km; ++u) C.aa[u] = 0.0;

  // integration, reversed
  int Lt = C.L[0];
  double Xt = C.x[0];
  for (int k2 = 0; k2 < kn; ++k2) {
    const int Lb = C.L[k2 + 1];
    const double Xb = C.x[k2 + 1];
    const double g = g2(k2);
    const bool inside = (Lb == Lt) || (Lb == Lt + 1 && Xb == 0.0);
    if (inside) {
      if (Xt == 0.0 && (Lb == Lt + 1 || Xb == 1.0)) C.qa[Lt] += g;
      else pmean_grad(Xt, Lb == Lt ? Xb : 1.0, g, C.pl[Lt], C.pr[Lt], C.p6[Lt]);
    } else {
      const double ma = fast_div(g, pe2(k2 + 1) - pe2(k2));
      if (Xt == 0.0) C.qa[Lt] += ma * C.h[Lt];
      else pmean_grad(Xt, 1.0, ma * (C.h[Lt] * (1.0 - Xt)), C.pl[Lt], C.pr[Lt], C.p6[Lt]);
      for (int m = Lt + 1; m < Lb; ++m) C.qa[m] += ma * C.h[m];
      if (Xb >= 1.0) C.qa[Lb] += ma * (C.h[Lb] * Xb);
      else if (Xb > 0.0) pmean_grad(0.0, Xb, ma * (C.h[Lb] * Xb), C.pl[Lb], C.pr[Lb], C.p6[Lb]);
    }
    Lt = Lb;
    Xt = Xb;
  }

  // layer parabolas, reversed
  for (int k = 0; k < km; ++k) {
    const double pl = C.pl[k], pr = C.pr[k], p6 = C.p6[k];
    if (pl == 0.0 && pr == 0.0 && p6 == 0.0) continue;
    const LayerDer D = layer_der<ODD>(k >= 2 && k <= km - 3, C.q[k], C.a[k], C.a[k + 1], C.d[k], iv, floor_v);
    double gL, gR, gd, gq = pl + pr;
    if (!D.low) {
      const double gl = fma(-3.0, p6, pl), gr = fma(-3.0, p6, pr);
      gL = D.l[0] * gl + D.r[0] * gr;
      gR = D.l[1] * gl + D.r[1] * gr;
      gd = D.l[2] * gl + D.r[2] * gr;
      gq -= gL + gR;
    } else {
      double J[3][4];
      layer_der_low(k, km, C.q[k], C.a[k], C.a[k + 1], C.d[k], iv, floor_v, J);
      gq = pl * J[0][0] + pr * J[1][0] + p6 * J[2][0];
      gL = pl * J[0][1] + pr * J[1][1] + p6 * J[2][1];
      gR = pl * J[0][2] + pr * J[1][2] + p6 * J[2][2];
      gd = pl * J[0][3] + pr * J[1][3] + p6 * J[2][3];
    }
    C.qa[k] += gq;
    C.aa[k] += gL;
    C.aa[k + 1] += gR;
    C.da[k] += gd;
  }
  // interfaces, reversed
  for (int u = 0; u <= km; ++u) {
    const double g = C.aa[u];
    if (g == 0.0) continue;
    const InterfaceDer D = interface_der<ODD>(u, km, iv, qf, hf, u >= 1 ? C.d[u - 1] : 0.0, u < km ? C.d[u] : 0.0);
    for (int s = 0; s < 3; ++s)
      if (D.q[s] != 0.0) C.qa[D.lo + s] += D.q[s] * g;
    if (D.inner) {
      C.da[u - 1] = fma(D.dl, g, C.da[u - 1]);
      C.da[u] = fma(D.dr, g, C.da[u]);
    }
  }
  // slopes, reversed
  for (int k = 1; k <= km - 2; ++k) {
    const double g = C.da[k];
    if (g == 0.0) continue;
    double p[3];
    slope4_grad<ODD>(C.q[k - 1], C.q[k], C.q[k + 1], C.h[k - 1], C.h[k], C.h[k + 1], p);
    for (int s = 0; s < 3; ++s) C.qa[k - 1 + s] = fma(p[s], g, C.qa[k - 1 + s]);
  }
}

// Every interior column and tracer of the state (thread per column and
// tracer): pressures from ptop = ak[0] and the running sum of dp, targets
// ak + bk ps.
template <bool ODD>
__global__ void __launch_bounds__(64) k_remap_ad_state(const double* q, const double* dp, const double* ak,
                                                       const double* bk, const double* q2_ad, double* q_ad,
                                                       PlaneGeom pg, long long P, int n, int nt, int nq, int km,
                                                       int kn, int iv, double floor_v, int* odd) {
  if (ODD && *odd == 0) return;
  const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long ncol = (long long)nt * n * n;
  if (id >= ncol * nq) return;
  const int iq = (int)(id / ncol);
  const long long col = id % ncol;
  const int t = (int)(col / ((long long)n * n));
  const int rem = (int)(col % ((long long)n * n));
  const int i = 1 + rem % n, j = 1 + rem / n;
  const long long p = pg.at(i, j);
  ColumnAd C;
  const long long qb = ((long long)t * nq + iq) * km * P + p;
  for (int k = 0; k < km; ++k) C.q[k] = q[qb + (long long)k * P];
  if (odd_column(C.q, km) != ODD) {
    if (!ODD) *odd = 1;
    return;
  }
  const double* dpc = dp + (long long)t * km * P + p;
  double ps = ak[0];
  for (int k = 0; k < km; ++k) ps += dpc[(long long)k * P];
  // pe1 as the forward kernel accumulates it (ptop, then + dp layer by layer)
  double pe1v[KMAX + 1];
  pe1v[0] = ak[0];
  for (int k = 0; k < km; ++k) pe1v[k + 1] = pe1v[k] + dpc[(long long)k * P];
  auto pe1 = [&](int k) { return pe1v[k]; };
  auto pe2 = [&](int k) { return ak[k] + bk[k] * ps; };
  const long long ob = ((long long)t * nq + iq) * kn * P + p;
  auto g2 = [&](int k2) { return q2_ad[ob + (long long)k2 * P]; };
  column_ad4<ODD>(C, km, kn, iv, floor_v, 0.0, pe1, pe2, g2);
  for (int k = 0; k < km; ++k) q_ad[qb + (long long)k * P] = C.qa[k];
}

// Tangent-linear of the same columns: the tangents of the slopes, interfaces and
// layers from their closed-form derivatives, integrated over the overlaps.
struct ColumnTl {
  static constexpr bool DUAL = true;
  double q[KMAX], h[KMAX], d[KMAX], a[KMAX + 1];
  double t[KMAX], td[KMAX], ta[KMAX + 1];  // tangents of the means, slopes and interfaces
  double tl[KMAX], tr[KMAX], t6[KMAX];     // and of the layer parabolas
};
template <bool ODD>
__global__ void __launch_bounds__(64) k_remap_tl4_state(const double* q, const double* dq, const double* dp,
                                                        const double* ak, const double* bk, double* dq2, PlaneGeom pg,
                                                        long long P, int n, int nt, int nq, int km, int kn, int iv,
                                                        double floor_v, int* odd) {
  if (ODD && *odd == 0) return;
  const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long ncol = (long long)nt * n * n;
  if (id >= ncol * nq) return;
  const int iq = (int)(id / ncol);
  const long long col = id % ncol;
  const int t = (int)(col / ((long long)n * n));
  const int rem = (int)(col % ((long long)n * n));
  const long long p = pg.at(1 + rem % n, 1 + rem / n);
  ColumnTl C;
  const long long qb = ((long long)t * nq + iq) * km * P + p;
  const double* dpc = dp + (long long)t * km * P + p;
  double ps = ak[0];
  for (int k = 0; k < km; ++k) {
    C.q[k] = q[qb + (long long)k * P];
    C.t[k] = dq[qb + (long long)k * P];
    const double next = ps + dpc[(long long)k * P];
    C.h[k] = next - ps;  // as the forward kernel: differences of the running pressure
    ps = next;
  }
  if (odd_column(C.q, km) != ODD) {
    if (!ODD) *odd = 1;
    return;
  }
  auto qf = [&](int k) -> double { return C.q[min(max(k, 0), km - 1)]; };
  auto hf = [&](int k) -> double { return C.h[min(max(k, 0), km - 1)]; };
  column_forward4<ODD>(C, km, iv, 0.0, qf, hf);
  for (int k = 0; k < km; ++k) {
    double g[3], v = 0.0;
    if (k >= 1 && k <= km - 2) {
      slope4_grad<ODD, true>(C.q[k - 1], C.q[k], C.q[k + 1], C.h[k - 1], C.h[k], C.h[k + 1], g);
      v = fma(g[0], C.t[k - 1], fma(g[1], C.t[k], g[2] * C.t[k + 1]));
    }
    C.td[k] = v;
  }
  for (int u = 0; u <= km; ++u) {
    const InterfaceDer D = interface_der<ODD>(u, km, iv, qf, hf, u >= 1 ? C.d[u - 1] : 0.0, u < km ? C.d[u] : 0.0);
    double v = 0.0;
    for (int s = 0; s < 3; ++s)
      if (D.q[s] != 0.0) v = fma(D.q[s], C.t[D.lo + s], v);
    if (D.inner) v += fma(D.dl, C.td[u - 1], D.dr * C.td[u]);
    C.ta[u] = v;
  }
  // a tangent that a branch leaves out (coefficient zero) may be NaN
  auto term = [](double c, double x) -> double { return nonzero(c) ? c * x : 0.0; };
  for (int k = 0; k < km; ++k) {
    const LayerDer D = layer_der<ODD>(k >= 2 && k <= km - 3, C.q[k], C.a[k], C.a[k + 1], C.d[k], iv, floor_v);
    if (!D.low) {
      const double eL = C.ta[k] - C.t[k], eR = C.ta[k + 1] - C.t[k];
      double bl = D.l[0] * eL + D.l[1] * eR + D.l[2] * C.td[k], br = D.r[0] * eL + D.r[1] * eR + D.r[2] * C.td[k];
      if (ODD) {
        bl = term(D.l[0], eL) + term(D.l[1], eR) + term(D.l[2], C.td[k]);
        br = term(D.r[0], eL) + term(D.r[1], eR) + term(D.r[2], C.td[k]);
      }
      C.tl[k] = C.t[k] + bl;
      C.tr[k] = C.t[k] + br;
      C.t6[k] = -3.0 * (bl + br);
    } else {
      double J[3][4];
      const bool finite = layer_der_low(k, km, C.q[k], C.a[k], C.a[k + 1], C.d[k], iv, floor_v, J);
      const double in[4] = {C.t[k], C.ta[k], C.ta[k + 1], C.td[k]};
      double o[3] = {0.0, 0.0, 0.0};
      for (int r = 0; r < 3; ++r)
        for (int s = 0; s < 4; ++s) o[r] += ODD ? term(J[r][s], in[s]) : J[r][s] * in[s];
      C.tl[k] = !ODD || finite ? o[0] : kNaN;
      C.tr[k] = !ODD || finite ? o[1] : kNaN;
      C.t6[k] = !ODD || finite ? o[2] : kNaN;
    }
  }
  // the overlaps, target by target; an infinity or a NaN in a layer makes its share NaN
  auto tan = [&](int k) -> double { return ODD && inf_or_nan(C.q[k]) ? kNaN : C.t[k]; };
  auto mean = [&](int k, double x1, double x2) {
    const double m = 0.5 * (x1 + x2);
    return C.tl[k] + m * ((C.tr[k] - C.tl[k]) + C.t6[k]) - C.t6[k] * ((x2 * x2 + x1 * x2 + x1 * x1) * (1.0 / 3.0));
  };
  const long long ob = ((long long)t * nq + iq) * kn * P + p;
  double lo = ak[0], hi = ak[0] + dpc[0], pe = ak[0] + bk[0] * ps;
  int k1 = 0;
  auto locate = [&](double pt) {
    while (k1 < km - 1 && !less(pt, hi)) {
      ++k1;
      lo = hi;
      hi = hi + dpc[(long long)k1 * P];
    }
    return fast_div(pt - lo, hi - lo);
  };
  double Xt = locate(pe);
  int Lt = k1;
  for (int k2 = 0; k2 < kn; ++k2) {
    const double pn = ak[k2 + 1] + bk[k2 + 1] * ps, Xb = locate(pn);
    const int Lb = k1;
    const bool inside = Lb == Lt || (Lb == Lt + 1 && Xb == 0.0);
    double out;
    if (inside) {
      out = Xt == 0.0 && (Lb == Lt + 1 || Xb == 1.0) ? C.t[Lt] : mean(Lt, Xt, Lb == Lt ? Xb : 1.0);
    } else {
      double m = Xt == 0.0 ? tan(Lt) * C.h[Lt] : (C.h[Lt] * (1.0 - Xt)) * mean(Lt, Xt, 1.0);
      for (int k = Lt + 1; k < Lb; ++k) m = fma(tan(k), C.h[k], m);
      if (Xb >= 1.0) m = fma(tan(Lb), C.h[Lb] * Xb, m);
      else if (Xb > 0.0) m = fma(C.h[Lb] * Xb, mean(Lb, 0.0, Xb), m);
      out = fast_div(m, pn - pe);
    }
    dq2[ob + (long long)k2 * P] = out;
    Lt = Lb;
    Xt = Xb;
    pe = pn;
  }
}

// One row of drop-in columns, [level][column] layout.
__global__ void __launch_bounds__(64) k_remap_ad_rows(const double* q1, const double* pe1, const double* pe2,
                                                      const double* qs, const double* q2_ad, double* q1_ad, int ncol,
                                                      int km, int kn, int iv) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= ncol) return;
  ColumnAd C;
  for (int k = 0; k < km; ++k) C.q[k] = q1[(long long)k * ncol + col];
  auto p1 = [&](int k) { return pe1[(long long)k * ncol + col]; };
  auto p2 = [&](int k) { return pe2[(long long)k * ncol + col]; };
  auto g2 = [&](int k2) { return q2_ad[(long long)k2 * ncol + col]; };
  column_ad4<true>(C, km, kn, iv, 0.0, qs ? qs[col] : 0.0, p1, p2, g2);
  for (int k = 0; k < km; ++k) q1_ad[(long long)k * ncol + col] += C.qa[k];
}

}  // namespace

namespace {
__global__ void k_pack_dual2(Dual<double>* out, const double* v, const double* d, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = Dual<double>(v[i], d ? d[i] : 0.0);
}
__global__ void k_unpack_tangent(const Dual<double>* in, double* d, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    d[i] = in[i].d;
}
unsigned blocks_for(long long n) { return (unsigned)std::min<long long>((n + 255) / 256, 8 * 152); }
}  // namespace

int lin_pack_dual(Dual<double>* out, const double* v, const double* d, long long n, cudaStream_t s) {
  k_pack_dual2<<<blocks_for(n), 256, 0, s>>>(out, v, d, n);
  FV3G_CUDA(cudaGetLastError());
  return 0;
}

int lin_unpack_tangent(const Dual<double>* in, double* d, long long n, cudaStream_t s) {
  k_unpack_tangent<<<blocks_for(n), 256, 0, s>>>(in, d, n);
  FV3G_CUDA(cudaGetLastError());
  return 0;
}

int lin_trajectory(const LinArgs& a, const double* q, const LinTraj& tr, cudaStream_t s) {
  const dim3 g = plane_grid(a);
  FV3G_CUDA(cudaMemsetAsync(a.odd, 0, sizeof(int), s));
  if (a.dr) k_lin_ratios<<<dim3(g.x, (unsigned)(a.nt * a.npz)), 128, 0, s>>>(a);
  k_lin_corners<<<g, 128, 0, s>>>(a, q, tr.qc1, tr.qc2);
  const int lines = std::max(a.ied - a.isd, a.jed - a.jsd) + 1;
  const dim3 ge((unsigned)((lines * 10 + 127) / 128), g.y, 2);
  const bool edges = a.ew != NO_EDGE || a.ee != NO_EDGE || a.es != NO_EDGE || a.en != NO_EDGE;
  k_lin_inner<<<g, 128, 0, s>>>(a, tr);
  if (edges) k_lin_edges<<<ge, 128, 0, s>>>(a, tr, 0);
  k_lin_odd<<<152 * 4, 128, 0, s>>>(a, tr, 0);
  k_lin_mid<<<g, 128, 0, s>>>(a, tr.qc1, tr.qc2, tr.fx2, tr.fy2, tr.qi, tr.qj);
  k_lin_outer<<<g, 128, 0, s>>>(a, tr);
  if (edges) k_lin_edges<<<ge, 128, 0, s>>>(a, tr, 1);
  k_lin_odd<<<152 * 4, 128, 0, s>>>(a, tr, 1);
  FV3G_CUDA(cudaGetLastError());
  return 0;
}

int lin_substep_tl(const LinArgs& a, const LinTraj& tr, const LinWork& w, const double* dq, double* dq_out,
                   cudaStream_t s) {
  const dim3 g = plane_grid(a);
  k_lin_corners<<<g, 128, 0, s>>>(a, dq, w.a1, w.a2);
  k_tl_inner<<<g, 128, 0, s>>>(a, tr, w.a1, w.a2, w.fx2, w.fy2);
  k_lin_mid<<<g, 128, 0, s>>>(a, w.a1, w.a2, w.fx2, w.fy2, w.ai, w.aj);
  k_tl_update<<<g, 128, 0, s>>>(a, tr, dq, w.ai, w.aj, w.fx2, w.fy2, dq_out);
  FV3G_CUDA(cudaGetLastError());
  return 0;
}

int lin_substep_ad(const LinArgs& a, const LinTraj& tr, const LinWork& w, const double* q_ad_out, double* q_ad_in,
                   cudaStream_t s) {
  const dim3 g = plane_grid(a);
  k_ad_faces<<<g, 128, 0, s>>>(a, q_ad_out, w.gx, w.gy);
  k_ad_outer<<<g, 128, 0, s>>>(a, tr, w.gx, w.gy, w.ai, w.aj);
  k_ad_mid<<<g, 128, 0, s>>>(a, w.ai, w.aj, w.gx, w.gy, w.fx2, w.fy2);
  k_ad_inner<<<g, 128, 0, s>>>(a, tr, w.ai, w.aj, w.fx2, w.fy2, w.a1, w.a2);
  // the collected adjoint goes through gx (free after k_ad_mid) before the halo transpose
  k_ad_collect<<<g, 128, 0, s>>>(a, q_ad_out, w.a1, w.a2, w.gx, 0);
  const long long nc = (long long)a.nt * a.nq * a.npz * 4;
  k_ad_corners<<<(unsigned)((nc + 127) / 128), 128, 0, s>>>(a, w.a1, w.a2, w.gx);
  k_ad_halo<<<g, 128, 0, s>>>(a, w.gx, q_ad_in);
  FV3G_CUDA(cudaGetLastError());
  return 0;
}

int lin_fluxes_ad(const LinArgs& a, const LinTraj& tr, const LinWork& w, const double* fx_ad, const double* fy_ad,
                  const double* d6x, const double* d6y, double* q_ad, cudaStream_t s) {
  const dim3 g = plane_grid(a);
  k_ad_flux_in<<<g, 128, 0, s>>>(a, fx_ad, fy_ad, w.gx, w.gy);
  k_ad_outer<<<g, 128, 0, s>>>(a, tr, w.gx, w.gy, w.ai, w.aj);
  k_ad_mid<<<g, 128, 0, s>>>(a, w.ai, w.aj, w.gx, w.gy, w.fx2, w.fy2);
  k_ad_inner<<<g, 128, 0, s>>>(a, tr, w.ai, w.aj, w.fx2, w.fy2, w.a1, w.a2);
  k_ad_collect<<<g, 128, 0, s>>>(a, nullptr, w.a1, w.a2, q_ad, 1);
  const long long nc = (long long)a.nt * a.nq * a.npz * 4;
  k_ad_corners<<<(unsigned)((nc + 127) / 128), 128, 0, s>>>(a, w.a1, w.a2, q_ad);
  if (d6x || d6y) k_ad_damp<<<g, 128, 0, s>>>(a, fx_ad, fy_ad, d6x, d6y, q_ad);
  FV3G_CUDA(cudaGetLastError());
  return 0;
}

LinArgs lin_state_args(const PlaneGeom& pg, long long P, int n, int nt, int nq, int npz, int hord, double lim_fac,
                       const Topo& topo) {
  LinArgs a{};
  a.pg = pg;
  a.P = P;
  a.is = 1; a.ie = n; a.js = 1; a.je = n;
  a.isd = 1 - NG; a.ied = n + NG; a.jsd = 1 - NG; a.jed = n + NG;
  a.npx = n + 1; a.npy = n + 1;
  a.ew = 1; a.ee = n + 1; a.es = 1; a.en = n + 1;
  a.corners = 15;
  a.n = n; a.nt = nt; a.nq = nq; a.npz = npz;
  a.hord = hord;
  a.lim_fac = lim_fac;
  a.topo = topo;
  return a;
}

int lin_remap_ad(const double* q, const double* dp, const double* ak, const double* bk, const double* q2_ad,
                 double* q_ad, PlaneGeom pg, long long P, int n, int nt, int nq, int km, int kn, int iv,
                 double q_min, int kord, int* odd, cudaStream_t s) {
  if (kord != 4) return set_error(FV3G_E_UNSUPPORTED, "the hand-written remap adjoint is kord 4 (got %d)", kord);
  if (km < 3 || km > KMAX || kn < 1 || kn > KMAX)
    return set_error(FV3G_E_ARG, "remap adjoint supports 3..%d layers (km=%d, kn=%d)", KMAX, km, kn);
  const long long nthr = (long long)nt * n * n * nq;
  FV3G_CUDA(cudaMemsetAsync(odd, 0, sizeof(int), s));
  for (auto kern : {k_remap_ad_state<false>, k_remap_ad_state<true>})  // the second: columns that the first reported
    kern<<<(unsigned)((nthr + 63) / 64), 64, 0, s>>>(q, dp, ak, bk, q2_ad, q_ad, pg, P, n, nt, nq, km, kn, iv,
                                                     iv == 1 ? q_min : 0.0, odd);
  FV3G_CUDA(cudaGetLastError());
  return 0;
}

int lin_remap_tl4(const double* q, const double* dq, const double* dp, const double* ak, const double* bk, double* dq2,
                  PlaneGeom pg, long long P, int n, int nt, int nq, int km, int kn, int iv, double q_min, int* odd,
                  cudaStream_t s) {
  if (km < 2 || km > KMAX || kn < 1 || kn > KMAX)
    return set_error(FV3G_E_ARG, "remap supports 2..%d layers (km=%d, kn=%d)", KMAX, km, kn);
  const long long nthr = (long long)nt * n * n * nq;
  FV3G_CUDA(cudaMemsetAsync(odd, 0, sizeof(int), s));
  for (auto kern : {k_remap_tl4_state<false>, k_remap_tl4_state<true>})
    kern<<<(unsigned)((nthr + 63) / 64), 64, 0, s>>>(q, dq, dp, ak, bk, dq2, pg, P, n, nt, nq, km, kn, iv,
                                                     iv == 1 ? q_min : 0.0, odd);
  FV3G_CUDA(cudaGetLastError());
  return 0;
}

int lin_remap_ad_rows(const double* q1, const double* pe1, const double* pe2, const double* qs, const double* q2_ad,
                      double* q1_ad, int ncol, int km, int kn, int iv, int kord, cudaStream_t s) {
  if (kord != 4) return set_error(FV3G_E_UNSUPPORTED, "the hand-written remap adjoint is kord 4 (got %d)", kord);
  if (km < 3 || km > KMAX || kn < 1 || kn > KMAX)
    return set_error(FV3G_E_ARG, "remap adjoint supports 3..%d layers (km=%d, kn=%d)", KMAX, km, kn);
  k_remap_ad_rows<<<(unsigned)((ncol + 63) / 64), 64, 0, s>>>(q1, pe1, pe2, qs, q2_ad, q1_ad, ncol, km, kn, iv);
  FV3G_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace fv3g
