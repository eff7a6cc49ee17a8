// fv3g_stream.cuh -- one tracer_2d substep (fv_tp_2d and the flux-form update)
// as a march along j.
//
// The body of tracer_2d's substep loop (fv_tracer2d.F90) with fv_tp_2d /
// xppm / yppm / copy_corners (tp_core.F90) of GFDL_atmos_cubed_sphere (absent
// submodule, .gitmodules:1-4), the schemes of fv3g_substep.cuh.
//
// A warp owns one tracer of a strip of columns (NC adjacent columns per lane,
// 32 NC - 6 of them outputs at most) and marches it row by row; the four PPM
// sweeps of a row advance together:
//   * y sweeps (inner on q, outer on q_j): the line of a column is a lane's own
//     rolling registers (slope -> interface -> deviations -> flux);
//   * x sweeps (inner on q of row m, outer on q_i of row m-4): neighbouring
//     cells by warp shuffles, every cell once.
// At iteration m the row m is loaded, its inner x flux gives q_j(m), the y
// sweeps reach face m-2 (q_i(m-3) and the final y flux), and the row m-4 takes
// its outer x flux and is written.  No intermediate leaves the registers, q is
// read once and written once, and only the strip's 3-column halo and the march's
// 7 rows of run-in are computed twice.
// The level's fields (Courant numbers, area and mass fluxes, areas, and the
// reciprocals and thickness ratios that k_level forms once for all tracers) are
// shared by the CTA's warps, one tracer each, through a ring of three batches of
// rows in shared memory, filled a batch ahead by 16-byte asynchronous copies of all
// threads; one barrier a batch.
//
// Bound: the FP64 pipe, which has 1/64 of the FP32 rate here.  What counts is the
// number of FP64 instructions per cell, so min, max, signs, comparisons, scaling by
// powers of two and the upwind choice run on bit patterns in the integer pipe (as
// FP64 instructions each takes 16 cycles of the SM), the flux is formed for the
// upwind cell only, what depends on the level alone is formed once for its tracers
// (k_level), and no cell but the strip's halo is swept twice; the windowed kernel
// (fv3g_substep.cuh) sweeps 1.5 cells per output cell and direction.  FP32 states,
// which instruction issue bounds, keep the windowed kernel: an FP32 form of this march took
// 6.1 ms at 6 x C192 L127 x 9 tracers and 11.2 at 6 x C384 L64 x 16, the windowed kernel
// 6.0 and 11.1 then and 4.5 at the former since.  Measured FP64, with the remap: a step of
// 6 x C192 L127 x 9 tracers, n_split 3, hord 8, 460 -> 172 ms, its substep 44 ms; of 6 x C96
// L64 x 4, 6 substeps, hord 5, 42.8 -> 18.3 ms, its substep 2.45 ms (FP64 pipe 84 % busy).
// Two columns a lane spill 56 bytes at hord 8 (255 registers).
#pragma once

#include <algorithm>
#include <type_traits>

#include "fv3g_fp64.cuh"
#include "fv3g_stencil.cuh"

namespace fv3g {

constexpr unsigned FULL = 0xffffffffu;

constexpr int SB = 4;            // rows per batch

// Strips and chunks of a launch: ns strips of W columns, nch chunks of H rows,
// ng groups of tracers (G per CTA, one warp each).
struct StreamMap {
  int ns, W, nch, H, ng, G;
};

enum { LX1 = 0, LX2, LXF, LAR, LMX, LY1, LY2, LYF, LMY, LDP, LRA, LRX, LRY, LN };
// Shared memory: the ring of level rows, each [field][column], the rows' edge
// weights (AdvArgs::ew), per warp q and the inner x flux of four rows, the fields' bases.
template <int NC>
struct StreamSmem {
  static constexpr int C = 32 * NC, ROW = LN * C;  // elements of a row
  double *rows, *ew, *hist;
  const double** base;
  __device__ __forceinline__ StreamSmem(unsigned char* raw, int warps) {
    rows = reinterpret_cast<double*>(raw);
    ew = rows + 3 * SB * ROW;
    hist = ew + 3 * SB * 8;
    base = reinterpret_cast<const double**>(hist + warps * 8 * C);
  }
  static size_t bytes(int warps) {
    return 8 * (size_t)(3 * SB * (ROW + 8) + warps * 8 * C) + LN * sizeof(double*);
  }
};

constexpr double kT11 = 11.0 / 14.0, kT14 = 4.0 / 7.0, kT15 = 3.0 / 14.0;  // hord 8 one-sided interfaces
constexpr double kD1 = -2.0 / 14.0, kD2 = 11.0 / 14.0, kD3 = 5.0 / 14.0;   // hord 1 / 5

// ------------------------------------------------------- lane vectors ---
// The NC columns of a lane.
template <int NC>
struct Vec {
  double v[NC];
  __device__ __forceinline__ double& operator[](int c) { return v[c]; }
  __device__ __forceinline__ const double& operator[](int c) const { return v[c]; }
};
template <int NC, class F>
__device__ __forceinline__ Vec<NC> vmap(F f) {
  Vec<NC> r;
#pragma unroll
  for (int c = 0; c < NC; ++c) r[c] = f(c);
  return r;
}
template <int NC>
__device__ __forceinline__ Vec<NC> operator+(const Vec<NC>& a, const Vec<NC>& b) {
  return vmap<NC>([&](int c) { return a[c] + b[c]; });
}
template <int NC>
__device__ __forceinline__ Vec<NC> operator-(const Vec<NC>& a, const Vec<NC>& b) {
  return vmap<NC>([&](int c) { return a[c] - b[c]; });
}
template <int NC>
__device__ __forceinline__ Vec<NC> operator*(const Vec<NC>& a, const Vec<NC>& b) {
  return vmap<NC>([&](int c) { return a[c] * b[c]; });
}
template <int NC>
__device__ __forceinline__ Vec<NC> vfma(const Vec<NC>& a, const Vec<NC>& b, const Vec<NC>& d) {
  return vmap<NC>([&](int c) { return fma(a[c], b[c], d[c]); });
}
template <int NC>
__device__ __forceinline__ Vec<NC> vzero() {
  return vmap<NC>([](int) { return 0.0; });
}
// values shifted by one column: of the column before (first: the lane before's last), of the column after
template <int NC>
__device__ __forceinline__ Vec<NC> vwest(const Vec<NC>& a) {
  Vec<NC> r;
  r[0] = __shfl_up_sync(FULL, a[NC - 1], 1);
  if (NC == 2) r[NC - 1] = a[0];
  return r;
}
template <int NC>
__device__ __forceinline__ Vec<NC> veast(const Vec<NC>& a) {
  Vec<NC> r;
  r[NC - 1] = __shfl_down_sync(FULL, a[0], 1);
  if (NC == 2) r[0] = a[NC - 1];
  return r;
}

// Monotonized central slopes in half increments: dm, |2 dm| and the sign; dp
// and d are the differences to the cells before and after.  Beside a NaN the slope is
// zero, as the minimum of the numbers left has it; that of an infinite cell is |xt| / 4, or, where
// xt is no finite number, the lesser of |d| and |dp|, infinite or NaN, as the bounds leave it.
template <int NC>
struct Slope {
  Vec<NC> dm, two;
  __device__ __forceinline__ void set(const Vec<NC>& xm, const Vec<NC>& x0, const Vec<NC>& xp, const Vec<NC>& dp,
                                      const Vec<NC>& d) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const double xt = xp[c] - xm[c];
      const bool odd = inf_or_nan(x0[c]);
      const bool mono = (__double2hiint(dp[c]) ^ __double2hiint(d[c])) >= 0 || odd;
      const double m = mag_min(quarter_mag(xt, odd), mag_min(absv(d[c]), absv(dp[c])));
      const double mag = mono ? m : 0.0;
      dm[c] = signed_as(mag, xt);
      two[c] = scale2<1>(mag);
    }
  }
  // edge deviations at most |2 dm| with the sign of dm (Lin 2004) from the raw
  // ones: nl the left one's negative, br the right one
  __device__ __forceinline__ void limit(const Vec<NC>& rl, const Vec<NC>& rr, Vec<NC>& nl,
                                        Vec<NC>& br) const {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      nl[c] = signed_as(mag_min(two[c], absv(rl[c])), dm[c]);
      br[c] = signed_as(mag_min(two[c], absv(rr[c])), dm[c]);
    }
  }
};

// Raw deviations d/2 + u/3 and -d/2 + u/3 of an interface from the cells before and
// after it: d their difference, u the difference of their slopes; halving is an
// exponent decrement.
template <int NC>
__device__ __forceinline__ void interface_raw(const Vec<NC>& d, const Vec<NC>& u, Vec<NC>& before, Vec<NC>& after) {
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const double h = scale2<-1>(d[c]);
    before[c] = fma(u[c], 1.0 / 3.0, h);
    after[c] = fma(u[c], 1.0 / 3.0, negv(h));
  }
}

// Courant numbers of a row's faces as the fluxes use them, from the planes that
// k_level forms: w1 = 1 - |c|, w2 = |c| (1 - |c|), and c > 0, which is carried by
// the sign of the stored w2 (that of w1 when c > 0, else the other one).
template <int NC>
struct FaceC {
  Vec<NC> w1, nw2;  // nw2 = -w2
  bool pos[NC];
  __device__ __forceinline__ void set(const Vec<NC>& a, const Vec<NC>& b) {
    w1 = a;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      pos[c] = (__double2hiint(a[c]) ^ __double2hiint(b[c])) >= 0;
      nw2[c] = pos[c] ? negv(b[c]) : b[c];
    }
  }
};

// x_up + w1 d_up - w2 b0_up of the upwind cell (left: xl, its right deviation
// br and b0; right: xr, the negative of its left deviation nl, and b0); keep
// false (hord 1, 5): the first-order upwind value
template <int HORD, int NC>
__device__ __forceinline__ Vec<NC> upwind(const FaceC<NC>& f, const Vec<NC>& xl, const Vec<NC>& br, const Vec<NC>& b0l,
                                          const Vec<NC>& xr, const Vec<NC>& nl, const Vec<NC>& b0r,
                                          const bool (&keep)[NC]) {
  return vmap<NC>([&](int c) {  // choose, then compute
    const double x = f.pos[c] ? xl[c] : xr[c], d = f.pos[c] ? br[c] : negv(nl[c]), b = f.pos[c] ? b0l[c] : b0r[c];
    const double v = fma(f.nw2[c], b, fma(f.w1[c], d, x));
    return HORD == 8 || keep[c] ? v : x;
  });
}

// 2-dx filter test of a cell (hord 5: bl br < 0; hord 1: |lim_fac b0| < |bl - br|); none
// beside a NaN passes
template <int HORD>
__device__ __forceinline__ bool filter_pass(double lim, double nl, double br, double b0) {
  if (HORD == 1) return dbits(absv(lim * b0)) < dbits(absv(nl + br)) && !is_nan(nl + br);
  return opp(negv(nl), br) && !is_nan(nl) && !is_nan(br);
}

// a linear form of four cells
__device__ __forceinline__ double form4(const double* w, double x2, double x1, double x0, double x3) {
  return fma(w[0], x2, fma(w[1], x1, fma(w[2], x0, w[3] * x3)));
}

// hord 8: raw deviations (of the cell before: rb, after: ra) of the interface
// between x1 and x0 beside a cube-face edge e: kind 1 interface e-1, 2 the edge, 3
// e+1; high: the tile lies below the edge.  x2, x3 the cells beyond x1 and x0, dm1
// and dm0 the slopes of x1 and x0.
__device__ __forceinline__ void edge_raw8(int kind, bool high, double x2, double x1, double x0, double x3, double dm1, double dm0, const double* w, double& rb,
                                          double& ra) {
  if (kind == 2) {
    const double a0 = clamp_between(form4(w, x2, x1, x0, x3), x1, x0);
    rb = a0 - x1;
    ra = a0 - x0;
  } else if (kind == 1) {
    if (high) {
      const double am = fma(kT14, dm1, fma(kT11, x1, kT15 * x0));
      rb = am - x1;
      ra = am - x0;
    } else {
      ra = fma(kT14, dm1, kT11 * (x1 - x0));
    }
  } else if (high) {
    rb = fma(-kT14, dm0, kT11 * (x0 - x1));
  } else {
    const double ap = fma(-kT14, dm0, fma(kT11, x0, kT15 * x1));
    rb = ap - x1;
    ra = ap - x0;
  }
}

// hord 1 / 5 interface between the second and third of four cells, by kind: 0 the
// fourth-order value, 1 and 3 the one-sided values beside a cube-face edge, 2 the
// edge value with weights w.  One form with weights chosen by kind costs four FP64
// instructions, as the fourth-order value alone does.
__device__ __forceinline__ double interface4(double x2, double x1, double x0, double x3) {
  return fma(7.0 / 12.0, x1 + x0, (-1.0 / 12.0) * (x2 + x3));
}
__device__ __forceinline__ double interface_edge(int kind, double x2, double x1, double x0, double x3,
                                                 const double* w) {
  double c[4];
  c[0] = kind == 2 ? w[0] : kind == 1 ? kD1 : kind == 3 ? 0.0 : -1.0 / 12.0;
  c[1] = kind == 2 ? w[1] : kind == 1 ? kD2 : kind == 3 ? kD3 : 7.0 / 12.0;
  c[2] = kind == 2 ? w[2] : kind == 1 ? kD3 : kind == 3 ? kD2 : 7.0 / 12.0;
  c[3] = kind == 2 ? w[3] : kind == 1 ? 0.0 : kind == 3 ? kD1 : -1.0 / 12.0;
  return form4(c, kind == 3 ? 0.0 : x2, x1, x0, kind == 1 ? 0.0 : x3);  // (0 times a NaN is one)
}

// CW84 eq. 1.10 with selects: 3 |d (bl + br)| > d^2, d = br - bl, as 3 |bl + br| > |d|.  Where
// bl br is NaN (bl + br is, or it is infinite beside a zero) the deviations stay.
__device__ __forceinline__ void cw84_flat(double& bl, double& br) {
  const double d = br - bl, s = bl + br;
  const bool zero = !nonzero(bl) || !nonzero(br);
  const bool odd = 2u * (unsigned)__double2hiint(s) > 0xffe00000u - zero;
  const bool big = mag_less(absv(d), absv(3.0 * s)) && !odd, down = (__double2hiint(d) ^ __double2hiint(s)) < 0;
  const double nl = big && down ? negv(scale2<1>(br)) : bl, nr = big && !down ? negv(scale2<1>(bl)) : br;
  const bool flat = (zero || (__double2hiint(bl) ^ __double2hiint(br)) >= 0) && !odd;
  bl = flat ? 0.0 : nl;
  br = flat ? 0.0 : nr;
}

// What a y march meets at its next face (row-uniform): the interface kind (1:
// e-1, 2: the cube-face edge e, 3: e+1, 0: none) and whether the cell it
// completes takes CW84 (hord 8).  high: the edge is the tile's north one.
struct RowSpec {
  int kind;
  bool high, cw;
};

// ------------------------------------------------------------ y line march ---
// The lines of the lane's columns.  Before step m the state holds x(m-3..m-1),
// and of cell m-2 the slope and left raw deviation (hord 8) or interface (hord
// 1, 5), and of cell m-3 the right deviation and b0; step(x(m)) returns the
// flux through face m-2.
template <int HORD, int NC>
struct YLine {
  using V = Vec<NC>;
  V xa, xb, xc, dp, rl, pbr, pb0;
  Slope<NC> sl;
  bool psm[NC];
  __device__ __forceinline__ void init() {
    xa = xb = xc = dp = rl = pbr = pb0 = vzero<NC>();
    sl.set(xa, xa, xa, xa, xa);
#pragma unroll
    for (int c = 0; c < NC; ++c) psm[c] = true;
  }
  template <bool SPEC>
  __device__ __forceinline__ V step(const V& x, const FaceC<NC>& f, double lim, const RowSpec& rs,
                                    const double (&dw)[NC][4]) {
    V nl, br, rn, b0;
    bool keep[NC];
    const V d = x - xc;
    if (HORD == 8) {
      Slope<NC> s1;
      s1.set(xb, xc, x, dp, d);  // cell m-1
      const V u = sl.dm - s1.dm;
      V rr;
      interface_raw(dp, u, rr, rn);  // interface m-1 less cell m-2 and less cell m-1
      if (SPEC && rs.kind != 0) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
          edge_raw8(rs.kind, rs.high, xa[c], xb[c], xc[c], x[c], sl.dm[c], s1.dm[c], dw[c], rr[c], rn[c]);
      }
      sl.limit(rl, rr, nl, br);
      if (SPEC && rs.cw) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          double l = rl[c], r = rr[c];
          cw84_flat(l, r);
          nl[c] = -l;
          br[c] = r;
        }
      }
      b0 = br - nl;
      sl = s1;
    } else {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        double al = interface4(xa[c], xb[c], xc[c], x[c]);
        if (SPEC && rs.kind != 0) al = interface_edge(rs.kind, xa[c], xb[c], xc[c], x[c], dw[c]);
        nl[c] = xb[c] - rl[c];  // rl: interface m-2
        br[c] = al - xb[c];
        rn[c] = al;
        b0[c] = br[c] - nl[c];
        const bool sm = filter_pass<HORD>(lim, nl[c], br[c], b0[c]);
        keep[c] = sm || psm[c];
        psm[c] = sm;
      }
    }
    const V fl = upwind<HORD, NC>(f, xa, pbr, pb0, xb, nl, b0, keep);
    xa = xb;
    xb = xc;
    xc = x;
    dp = d;
    rl = rn;
    pbr = br;
    pb0 = b0;
    return fl;
  }
};

// ------------------------------------------------------------ x line of a row ---
// What a lane's columns are to the cube-face edges: the kinds of the interfaces
// west of its columns, which of its cells take CW84, and which edge (0 west, 1
// east) that is.
template <int NC>
struct LaneEdge {
  int kind[NC];
  bool cw[NC];
  int side;
  bool face, any;
};

// Fluxes through the west faces of the lane's columns.
template <int HORD, int NC, bool EDGES>
__device__ __forceinline__ Vec<NC> x_line(const Vec<NC>& x, const FaceC<NC>& f, double lim,
                                             const LaneEdge<NC>& le, const double* dw) {
  using V = Vec<NC>;
  const V xm = vwest(x), xp = veast(x);
  V nl, br, b0;
  bool keep[NC];
  if (HORD == 8) {
    V d, de;  // differences across the west and the east interfaces
#pragma unroll
    for (int c = 0; c < NC; ++c) d[c] = x[c] - xm[c];
#pragma unroll
    for (int c = 0; c < NC; ++c) de[c] = c + 1 < NC ? d[c + 1 < NC ? c + 1 : 0] : xp[NC - 1] - x[NC - 1];
    Slope<NC> s;
    s.set(xm, x, xp, d, de);
    const V dmw = vwest(s.dm);
    V rl, rw;  // the west interfaces less the cell and less the cell west of it
    interface_raw(d, dmw - s.dm, rw, rl);
    if constexpr (EDGES) {
      const double x2w = NC == 1 ? __shfl_up_sync(FULL, x[0], 2) : __shfl_up_sync(FULL, x[0], 1);
      if (le.face) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
          if (le.kind[c] != 0)
            edge_raw8(le.kind[c], le.side == 1, c ? xm[c ? c - 1 : 0] : x2w, xm[c], x[c], xp[c], dmw[c], s.dm[c],
                      dw + le.side * 4, rw[c], rl[c]);
      }
      __syncwarp();
    }
    const V rr = veast(rw);
    s.limit(rl, rr, nl, br);
    if constexpr (EDGES) {
      if (le.any) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          double l = rl[c], r = rr[c];
          cw84_flat(l, r);
          nl[c] = le.cw[c] ? -l : nl[c];
          br[c] = le.cw[c] ? r : br[c];
        }
      }
      __syncwarp();
    }
    b0 = br - nl;
  } else {
    const double xw = NC == 1 ? __shfl_up_sync(FULL, x[0], 2) : __shfl_up_sync(FULL, x[0], 1);
    V al;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const double x2 = c ? xm[c ? c - 1 : 0] : xw;
      al[c] = EDGES ? interface_edge(le.kind[c], x2, xm[c], x[c], xp[c], dw + le.side * 4)
                    : interface4(x2, xm[c], x[c], xp[c]);
    }
    const V ae = veast(al);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      nl[c] = x[c] - al[c];
      br[c] = ae[c] - x[c];
      b0[c] = br[c] - nl[c];
    }
    int sm[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) sm[c] = filter_pass<HORD>(lim, nl[c], br[c], b0[c]);
    const int smw = __shfl_up_sync(FULL, sm[NC - 1], 1);
#pragma unroll
    for (int c = 0; c < NC; ++c) keep[c] = (sm[c] | (c ? sm[c ? c - 1 : 0] : smw)) != 0;
  }
  return upwind<HORD, NC>(f, xm, vwest(br), vwest(b0), x, nl, b0, keep);
}

// NC adjacent values of a row
template <int NC>
__device__ __forceinline__ void ld_row(const double* p, Vec<NC>& v) {
  if constexpr (NC == 1) {
    v[0] = p[0];
  } else {
    const double2 u = *reinterpret_cast<const double2*>(p);
    v[0] = u.x;
    v[1] = u.y;
  }
}
template <int NC>
__device__ __forceinline__ void st_row(double* p, const Vec<NC>& v) {
  if constexpr (NC == 1) p[0] = v[0];
  else *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
}
// 16 bytes into shared memory by an asynchronous copy
__device__ __forceinline__ void copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// ------------------------------------------------------------ the kernel ---
template <int HORD, int NC, bool EDGES>
struct March {
  using V = Vec<NC>;
  static constexpr int C = 32 * NC, ROW = LN * C;
  const AdvArgs<double>& a;
  int i0, j0, ni, nj;         // first output cell and size of the strip chunk
  int eS, eN;                 // window rows of the cube-face edges, or NO_EDGE
  int iq, lane;
  double lim;
  LaneEdge<NC> le;
  // rolling state
  YLine<HORD, NC> yi, yo;
  V qi;          // q_i(m-4)
  V fyy;         // yfx times the inner y flux of face m-3
  V Fp, Fy;      // final y fluxes (doubled) of faces m-4 and m-3
  V nx[2];       // rows m, m+1 in flight
  const double* qp;   // this lane's columns of row m+2
  double* op;         // of the row m-4

  // Row m of the march.  SPEC: any row (the run-in, rows beside a cube-face
  // edge or beyond it, the last ones); else an ordinary row with m >= 8.
  // r: the row's place in its pair of rows; p0, p1, p2: the lane's columns of array
  // 0 of this pair's level rows and the two pairs before, e0, e2 their edge weights.
  template <bool SPEC, int r>
  __device__ __forceinline__ void row(int m, const double* p0, const double* p1, const double* p2, const double* e0, const double* e2, double* hist) {
    const PlaneGeom& pg = a.pg;
    const int j = j0 - 3 + m, t = blockIdx.z, k = blockIdx.y;
    // edge-flux index (((t*4 + e)*npz + k)*nq + iq)*n + s = efo + e*efe + iq*n + s
    const long long efe = (long long)a.npz_e * a.nq * (a.npx - 1);
    const long long efo = (((long long)t * 4) * a.npz_e + k) * a.nq * (a.npx - 1);
    auto lev = [&](int arr, int back) -> V {  // array arr at row m - back
      V v;
      const int rr = r - back + 4;  // 0..5: rows of the pairs p2, p1, p0
      ld_row<NC>((rr < 2 ? p2 : rr < 4 ? p1 : p0) + (rr & 1) * ROW + arr * C, v);
      return v;
    };
    V x = nx[r], qy;
    if (!SPEC || m + 2 < nj + 6) ld_row<NC>(qp, nx[r]);  // row m + 2
    qp += pg.pitch;
    qy = x;
    if (SPEC) {
      // corner blocks: the copy_corners rotation of each sweep's direction
      if (!a.nested && a.corners != 0 && (j < 1 || j > a.npy - 1) && m < nj + 6) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const int i = i0 - 3 + lane * NC + c;
          if (i < 1 || i > a.npx - 1) {
            x[c] = load_q(a, t, iq, k, i, j, 1);
            qy[c] = load_q(a, t, iq, k, i, j, 2);
          }
        }
        __syncwarp();
      }
    }
    // ---- x sweeps: inner on row m, outer on q_i of row m-4
    FaceC<NC> fc;
    fc.set(lev(LX1, 0), lev(LX2, 0));
    const V fx2 = x_line<HORD, NC, EDGES>(x, fc, lim, le, e0 + r * 8);
    const V fxx = lev(LXF, 0) * fx2;
    const V qj = (vfma(x, lev(LAR, 0), fxx) - veast(fxx)) * lev(LRX, 0);
    V q4, f4;  // q and the inner x flux of row m-4, whose place row m takes
    ld_row<NC>(hist + r * 2 * C, q4);
    ld_row<NC>(hist + r * 2 * C + C, f4);
    st_row<NC>(hist + r * 2 * C, x);
    st_row<NC>(hist + r * 2 * C + C, fx2);
    if (!SPEC || m >= 7) {
      fc.set(lev(LX1, 4), lev(LX2, 4));
      const V fo = x_line<HORD, NC, EDGES>(qi, fc, lim, le, e2 + r * 8);
      const V F = (fo + f4) * lev(LMX, 4);
      if (EDGES && a.eflux != nullptr && m - 7 < nj) {  // outward fluxes through the tile's edges
        const int n = a.npx - 1, jr = j - 4;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const int i = i0 - 3 + lane * NC + c;
          if (i == 1 && i0 == 1) a.eflux[efo + iq * (long long)n + (jr - 1)] = double(-0.5) * F[c];
          if (i == a.npx && i == i0 + ni) a.eflux[efo + efe + iq * (long long)n + (jr - 1)] = double(0.5) * F[c];
        }
      }
      const V v = ((vfma(q4, lev(LDP, 4), F - veast(F)) + Fp) - Fy) * lev(LRA, 4);
      const int w = lane * NC - 3;  // output column of the lane's first
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (w + c >= 0 && w + c < ni && (!SPEC || m - 7 < nj)) op[c] = v[c];
      op += pg.pitch;
    }
    // ---- y sweeps to face m-2: q_i(m-3) and the final y flux
    RowSpec rs{0, false, false};
    double dw[NC][4];
    if (SPEC) {
      const int f = m - 1, cell = m - 2;  // window rows of the next interface and of the cell completed
      rs.kind = eS != NO_EDGE && f >= eS - 1 && f <= eS + 1 ? f - eS + 2
                : eN != NO_EDGE && f >= eN - 1 && f <= eN + 1 ? f - eN + 2 : 0;
      rs.high = !(eS != NO_EDGE && f <= eS + 1);
      rs.cw = (eS != NO_EDGE && cell >= eS - 1 && cell <= eS + 1) || (eN != NO_EDGE && cell >= eN - 2 && cell <= eN);
      if (rs.kind == 2) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const double* dya = a.dya + t * a.sMt;
          const int i = i0 - 3 + lane * NC + c, je = j0 - 3 + f;
          const double d2 = ld_field(dya, pg, i, je - 2), d1 = ld_field(dya, pg, i, je - 1), d0 = ld_field(dya, pg, i, je),
                  d3 = ld_field(dya, pg, i, je + 1);
          const double wl = d1 / (d1 + d2), wr = d0 / (d0 + d3);
          dw[c][0] = -0.5 * wl;
          dw[c][1] = 0.5 + 0.5 * wl;
          dw[c][2] = 0.5 + 0.5 * wr;
          dw[c][3] = -0.5 * wr;
        }
      }
    }
    FaceC<NC> fy;
    fy.set(lev(LY1, 2), lev(LY2, 2));
    const V q3 = yi.xa;  // q(m-3): its corner cells, which differ from the x sweeps', are not used
    const V fi = yi.template step<SPEC>(qy, fy, lim, rs, dw);
    const V fq = yo.template step<SPEC>(qj, fy, lim, rs, dw);
    const V g = lev(LYF, 2) * fi;
    qi = (vfma(q3, lev(LAR, 3), fyy) - g) * lev(LRY, 3);
    fyy = g;
    const V F = (fq + fi) * lev(LMY, 2);
    Fp = Fy;
    Fy = F;
    if (SPEC && a.eflux != nullptr) {
      const int n = a.npx - 1, jf = j - 2;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int i = i0 - 3 + lane * NC + c, w = lane * NC + c - 3;
        if (w < 0 || w >= ni) continue;
        if (jf == 1 && j0 == 1 && m >= 5) a.eflux[efo + 2 * efe + iq * (long long)n + (i - 1)] = double(-0.5) * Fy[c];
        if (jf == a.npy && m - 5 == nj) a.eflux[efo + 3 * efe + iq * (long long)n + (i - 1)] = double(0.5) * Fy[c];
      }
    }
  }
};

// One strip chunk of one tracer per warp.  EDGES: the strip's columns reach a
// cube-face edge.
template <int HORD, int NC, bool EDGES>
__device__ __forceinline__ void stream_body(const AdvArgs<double>& a, const StreamMap& sm, const StreamSmem<NC>& S, int strip,
                                            int group, int chunk, int eW, int eE) {
  constexpr int C = 32 * NC, ROW = LN * C;
  const PlaneGeom& pg = a.pg;
  const int tid = threadIdx.x, nth = blockDim.x;
  March<HORD, NC, EDGES> M{a};
  M.i0 = a.is + strip * sm.W;
  M.j0 = a.js + chunk * sm.H;
  M.ni = min(sm.W, a.ie - M.i0 + 1);
  M.nj = min(sm.H, a.je - M.j0 + 1);
  M.lane = tid & 31;
  M.iq = group * sm.G + (tid >> 5);
  const bool mine = M.iq < a.nq;  // a surplus warp of the last group only stages the level's rows
  M.lim = double(a.lim_fac);
  const int i0 = M.i0, j0 = M.j0, nj = M.nj, t = blockIdx.z, k = blockIdx.y;
  // window rows of the cube-face edges (cell e is the first beyond a low edge)
  M.eS = (!a.nested && a.js == 1 && j0 - 3 <= 3) ? 4 - j0 : NO_EDGE;
  M.eN = (!a.nested && a.je + 1 == a.npy && a.npy - j0 + 3 <= nj + 8) ? a.npy - j0 + 3 : NO_EDGE;
  M.le.any = M.le.face = false;
  M.le.side = 0;
  if (EDGES) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int w = M.lane * NC + c;
      M.le.kind[c] = 0;
      if (eW != NO_EDGE && w >= eW - 1 && w <= eW + 1) M.le.kind[c] = w - eW + 2;
      if (eE != NO_EDGE && w >= eE - 1 && w <= eE + 1) {
        M.le.kind[c] = w - eE + 2;
        M.le.side = 1;
      }
      M.le.cw[c] = (eW != NO_EDGE && w >= eW - 1 && w <= eW + 1) || (eE != NO_EDGE && w >= eE - 2 && w <= eE);
      M.le.any = M.le.any || M.le.cw[c];
      M.le.face = M.le.face || M.le.kind[c] != 0;
    }
  }
  // ---- level rows
  const long long fo = t * a.sFt + k * a.sFk, mo = t * a.sMt, lo = t * a.sLt + k * a.sFk;
  const int wof = i0 - 3 - pg.isd;  // plane column of window column 0 (a multiple of 16 bytes)
  const int nb = (nj + 7 + SB - 1) / SB;
  if (tid < LN) {
    const double* p = a.cx1 + lo;
    p = tid == LX2 ? a.cx2 + lo : p;
    p = tid == LXF ? a.xfx + fo : p;
    p = tid == LAR ? a.area + mo : p;
    p = tid == LMX ? a.mfx + fo : p;
    p = tid == LY1 ? a.cy1 + lo : p;
    p = tid == LY2 ? a.cy2 + lo : p;
    p = tid == LYF ? a.yfx + fo : p;
    p = tid == LMY ? a.mfy + fo : p;
    p = tid == LDP ? a.dpa + lo : p;
    p = tid == LRA ? a.ub + lo : p;
    p = tid == LRX ? a.rrx + lo : p;
    p = tid == LRY ? a.rry + lo : p;
    S.base[tid] = p + wof;
  }
  __syncthreads();
  auto copy_batch = [&](int bt, int slot) {
    // a warp copies RW rows of a field at a time: E elements per copy, CH copies per row
    constexpr int E = 16 / 8, CH = C / E, RW = 32 / CH;
    const int p = (M.lane % CH) * E, r0 = M.lane / CH;
    const int jb = j0 - 3 + bt * SB - pg.jsd, col = min(p, pg.pitch - wof - E);
    double* const dst = S.rows + slot * (SB * ROW) + p;
#pragma unroll 1
    for (int r = r0; r < SB; r += RW) {
      const int off = min(jb + r, pg.rows - 1) * pg.pitch + col;
#pragma unroll 1
      for (int arr = tid >> 5; arr < LN; arr += nth >> 5) copy16(dst + r * ROW + arr * C, S.base[arr] + off);
    }
    if (EDGES) {
      constexpr int EW = 8 / E;
      for (int e = tid; e < SB * EW; e += nth) {
        const int jr = min(jb + e / EW, pg.rows - 1);
        copy16(S.ew + slot * (SB * 8) + e * E, a.ew + ((long long)t * pg.rows + jr) * 8 + (e % EW) * E);
      }
    }
  };
  // ---- the march
  {
    const long long qb = t * a.sQt + M.iq * a.sQq + k * a.sQk;
    const int col = wof + M.lane * NC;
    const int cl = min(col, pg.pitch - NC);
    M.qp = a.q_in + qb + (long long)(j0 - 3 - pg.jsd) * pg.pitch + cl;
    M.op = a.q_out + qb + (long long)(j0 - pg.jsd) * pg.pitch + col;
    if (mine) {
      ld_row<NC>(M.qp, M.nx[0]);
      ld_row<NC>(M.qp + pg.pitch, M.nx[1]);
    }
    M.qp += 2 * pg.pitch;
  }
  M.yi.init();
  M.yo.init();
  M.qi = M.fyy = M.Fy = M.Fp = vzero<NC>();
  double* const hist = S.hist + (tid >> 5) * (8 * C) + M.lane * NC;  // this lane's columns of the last four rows
  copy_batch(0, 0);
  int slot = 0, before = 2;  // of batch bt and of the one before it
#pragma unroll 1
  for (int bt = 0; bt < nb; ++bt) {
    stage_wait();
    __syncthreads();  // batch bt has arrived; nobody reads the batch before the last one any more
    const int next = slot == 2 ? 0 : slot + 1;
    if (bt + 1 < nb) copy_batch(bt + 1, next);
    const int m0 = bt * SB;
    // the run-in, rows beside a cube-face edge of the tile and halo rows beyond it, and the last rows
    const bool spec = m0 < 8 || m0 + SB + 2 > nj + 6 || (M.eS != NO_EDGE && m0 <= M.eS + 3) ||
                      (M.eN != NO_EDGE && m0 + SB > M.eN) ||
                      (!a.nested && a.corners != 0 && j0 - 3 + m0 + SB - 1 > a.npy - 1);
    if (mine) {
      const double *const cur = S.rows + slot * (SB * ROW) + M.lane * NC, *const pre = S.rows + before * (SB * ROW) + M.lane * NC;
      const double *const ecur = S.ew + slot * (SB * 8), *const epre = S.ew + before * (SB * 8);
#pragma unroll 1
      for (int h = 0; h < SB; h += 2) {
        static_assert(SB == 4, "the rows four back are the same rows of the batch before");
        const int m = m0 + h;
        const double *p0 = cur + h * ROW, *p1 = h ? p0 - 2 * ROW : pre + 2 * ROW, *p2 = pre + h * ROW;
        const double *e0 = ecur + h * 8, *e2 = epre + h * 8;
        double* const pt = hist + (h & 2) * (2 * C);
        if (spec) {
          M.template row<true, 0>(m, p0, p1, p2, e0, e2, pt);
          M.template row<true, 1>(m + 1, p0, p1, p2, e0, e2, pt);
        } else {
          M.template row<false, 0>(m, p0, p1, p2, e0, e2, pt);
          M.template row<false, 1>(m + 1, p0, p1, p2, e0, e2, pt);
        }
      }
    }
    before = slot;
    slot = next;
  }
}

template <int HORD, int NC>
__global__ void __launch_bounds__(32 * STREAM_MAX_WARPS, 1) k_stream(const AdvArgs<double> a, const StreamMap sm) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const StreamSmem<NC> S(smem_raw, sm.G);
  int b = blockIdx.x;
  const int strip = b % sm.ns;
  b /= sm.ns;
  const int group = b % sm.ng, chunk = b / sm.ng;
  const int i0 = a.is + strip * sm.W;
  // window columns of the cube-face edges
  const int eW = (!a.nested && a.is == 1 && i0 - 3 <= 3) ? 4 - i0 : NO_EDGE;
  const int eE = (!a.nested && a.ie + 1 == a.npx && a.npx - i0 + 3 <= 32 * NC + 1) ? a.npx - i0 + 3 : NO_EDGE;
  if (eW != NO_EDGE || eE != NO_EDGE) stream_body<HORD, NC, true>(a, sm, S, strip, group, chunk, eW, eE);
  else stream_body<HORD, NC, false>(a, sm, S, strip, group, chunk, eW, eE);
}

// Strips, chunks and tracer groups of a launch.  Columns per lane: the choice
// that sweeps fewer lanes over the tile's width (32 NC per strip), one on a tie: twice
// the warps for the same FP64 work hide more of a row's latency and balance the SMs
// better (one face of C48 L63 x 1 492 to 381 us a step, six C192 L127 x 9 173 to 171 ms).
// It depends on the width alone, and the file is built without automatic contraction of
// products and sums (the fused ones are written), so that a cell's value does not depend on the
// chunk, and a tracer's result not on the batch, it is computed in.
inline int stream_columns(int ni) {
  const int two = ni <= 58 ? 64 : 64 * ((ni + 55) / 56), one = ni <= 26 ? 32 : 32 * ((ni + 23) / 24);
  return one <= two ? 1 : 2;
}

// Tracers per CTA and chunks along j, from a model of the launch: an SM holds
// res CTAs (registers: 255 a thread; shared memory), and with w warps resident a
// row of each takes time in proportion to w + c (the FP64 pipe shared, plus the
// latency of a row: c = 1.5 with two columns a lane, 83 % of the pipe used at 8 warps;
// 3 with one, whose row is half the work; 1.5 there took 381 us, 3 to 8 325 us, for one face of
// C48 L63 x 1).  A CTA pays for staging a
// row what one more tracer would cost in part (1 / G), a chunk 9 rows of run-in,
// and the launch whole waves of CTAs.  At six C192 tiles x 127 levels x 9 tracers
// groups of 3 and 5 took 52.9 and 59.8 ms a substep, at 4 tracers groups of 4 and 2
// 25.2 and 26.8 ms.
template <int NC>
inline StreamMap stream_map(int ni, int nj, int nq, int warps, long long planes) {
  StreamMap best{};
  // several strips start at multiples of 4 columns (16 bytes)
  const int most = 32 * NC - 6;
  best.ns = ni <= most ? 1 : (ni + (most & ~3) - 1) / (most & ~3);
  best.W = ((ni + best.ns - 1) / best.ns + 3) & ~3;
  best.ns = (ni + best.W - 1) / best.W;
  const int by_regs = 8;  // warps of an SM
  const double c = NC == 1 ? 3.0 : 1.5;
  double least = 0.0;
  for (int g = std::min(std::min(warps, STREAM_MAX_WARPS), nq); g >= 1; --g) {
    const int ng = (nq + g - 1) / g, G = (nq + ng - 1) / ng;
    const long long res = std::max<long long>(
        1, std::min<long long>(by_regs / G, (227 << 10) / (long long)(StreamSmem<NC>::bytes(G) + 1024)));
    for (int nch = 1; nch == 1 || nj / nch >= 8; ++nch) {
      const int H = (nj + nch - 1) / nch;
      const long long ctas = planes * best.ns * ng * ((nj + H - 1) / H), waves = (ctas + 152 * res - 1) / (152 * res);
      const double w = (double)G * (double)std::min(res, (ctas + 151) / 152);
      const double cost = (double)waves * (H + 9) * (w + c) * (1.0 + 1.0 / G);
      if (least == 0.0 || cost < 0.98 * least) {  // wider groups and fewer chunks unless clearly slower
        least = cost;
        best.ng = ng;
        best.G = G;
        best.H = H;
        best.nch = (nj + H - 1) / H;
      }
      if (waves > 8) break;  // enough CTAs
    }
  }
  return best;
}

template <int HORD, int NC>
int launch_stream_nc(const AdvArgs<double>& a, int warps, cudaStream_t s) {
  const int nt = adv_tiles(a);
  const StreamMap m =
      stream_map<NC>(a.ie - a.is + 1, a.je - a.js + 1, a.nq, std::max(warps, 1), (long long)nt * a.npz);
  dim3 grid((unsigned)(m.ns * m.ng * m.nch), a.npz, nt);
  k_stream<HORD, NC><<<grid, 32 * m.G, StreamSmem<NC>::bytes(m.G), s>>>(a, m);
  FV3G_CUDA(cudaGetLastError());
  return 0;
}

template <int HORD>
int launch_stream_h(const AdvArgs<double>& a, int warps, cudaStream_t s) {
  return stream_columns(a.ie - a.is + 1) == 2 ? launch_stream_nc<HORD, 2>(a, warps, s)
                                              : launch_stream_nc<HORD, 1>(a, warps, s);
}

template <int HORD>
void prepare_stream_h(cudaError_t& err) {
  const cudaError_t es[] = {cudaFuncSetAttribute(k_stream<HORD, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)StreamSmem<1>::bytes(STREAM_MAX_WARPS)),
                            cudaFuncSetAttribute(k_stream<HORD, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)StreamSmem<2>::bytes(STREAM_MAX_WARPS))};
  for (cudaError_t e : es)
    if (e != cudaSuccess && err == cudaSuccess) err = e;
}

}  // namespace fv3g

#define FV3G_STREAM_INSTANTIATE(H)                                             \
  namespace fv3g {                                                            \
  template int launch_stream_h<H>(const AdvArgs<double>&, int, cudaStream_t); \
  template void prepare_stream_h<H>(cudaError_t&);                            \
  }
