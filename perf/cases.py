"""The measured workloads of the tracer path: what a model that transports its tracers with this library has it do.

``listed()`` names them, ``draw(rng)`` gives more of the same ranges, ``prepare(case, seed)`` builds what a program
holds before the call (grid, levels, state, this step's fields), ``run(state)`` is one call through the public entry
points and ``exact(case, seed)`` restates the schemes in plain torch in 64 bits.  A pass starts from the step's own
inputs every time (the device-resident entries take them from device arrays, as a model on the GPU hands them over),
so every pass of one state computes the same thing.

Kinds of work:
  step      CubeState: upload the step's fields from device arrays, tracer_2d + remap as one call, the tracers out
  ensemble  members of several sizes advanced by one Ensemble call
  lin       tangent-linear or adjoint of a whole step about a resident trajectory (data assimilation)
  fields    the pt, u and v remaps beside the tracers
  host      one step from page-locked host arrays to host arrays
  dropin    tracer_2d and map_scalar_3d on a rank's own host arrays, the Fortran entries
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from fv3atm_gb300 import api
from fv3atm_gb300 import grid as G
from fv3atm_gb300 import synth as S

NG = 3
DEV = "cuda"


# ------------------------------------------------------------------- cases ---
def _step(name, n, npz, nq, *, tiles=6, indep=False, precision="mixed", hord=8, kord=9, split=3, nord=0, trdm=0.0,
          fill=False, mass_fix=False):
    c = dict(kind="step", n=n, npz=npz, nq=nq, tiles=tiles, indep=indep, precision=precision, hord=hord, kord=kord,
             split=split, nord=nord, trdm=trdm, fill=fill, mass_fix=mass_fix)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one C48 face with a prescribed halo ring and one tracer, the test-bed of the scheme: latency and launches
        _step("tile_c48_l63_q1_fp64", 48, 63, 1, tiles=1, precision="fp64", split=2),
        # a small ragged cube with the options a namelist turns on: del-4 damping, fillz, the mass fixer, and the
        # substep count derived from the winds (q_split 0)
        _step("cube_c45_l33_q3_options", 45, 33, 3, split=0, nord=1, trdm=0.02, fill=True, mass_fix=True),
        # an ensemble of single-face members of three sizes, advanced together
        dict(name="ensemble_c48_c96_c192_q4", kind="ensemble", members="48x32x16,96x64x10,192x127x6", nq=4, split=2),
        # the forward step of the linearised configuration, hord 5 / kord 4 in FP64
        _step("cube_c96_l64_q4_fp64_h5k4", 96, 64, 4, precision="fp64", hord=5, kord=4, split=6),
        # the standard global step in both precisions
        _step("cube_c192_l127_q9_mixed", 192, 127, 9),
        _step("cube_c192_l127_q9_fp64", 192, 127, 9, precision="fp64"),
        # the high-resolution global step with the full tracer list
        _step("cube_c384_l127_q20_mixed", 384, 127, 20),
        # tangent-linear and adjoint of a six-substep step
        dict(name="tl_c96_l64_q4", kind="lin", mode="tl", n=96, npz=64, nq=4, hord=5, kord=4, split=6),
        dict(name="ad_c96_l64_q4", kind="lin", mode="ad", n=96, npz=64, nq=4, hord=5, kord=4, split=6),
        # pt and the winds remapped beside the tracers
        dict(name="fields_c192_l127_mixed", kind="fields", n=192, npz=127, precision="mixed"),
        # a CPU model that hands its host arrays over every step
        dict(name="host_c192_l127_q9", kind="host", n=192, npz=127, nq=9, split=3),
        # one MPI rank's drop-in calls on a whole face
        dict(name="dropin_c48_l63_q3", kind="dropin", n=48, npz=63, nq=3, hord=8, kord=9, split=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "ensemble", "lin", "fields", "host", "dropin"])
    npz = rng.randint(12, 127)
    if kind == "step":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        n = _log_int(rng, 20, 288 if precision == "mixed" else 144)
        nq = _log_int(rng, 1, 20 if n < 200 else 12)
        one = rng.random() < 0.3
        tiles = rng.randint(1, 8) if one else 6
        hord, kord = rng.choice([(8, 9), (8, 9), (8, 4), (5, 9), (5, 4)])
        damp = rng.random() < 0.2
        return _step(None, n, npz, nq, tiles=tiles, indep=one, precision=precision, hord=hord, kord=kord,
                     split=rng.randint(1, 4), nord=rng.randint(0, 2) if damp else 0, trdm=0.02 if damp else 0.0,
                     fill=rng.random() < 0.2, mass_fix=rng.random() < 0.2)
    if kind == "ensemble":
        members = ",".join("%dx%dx%d" % (_log_int(rng, 24, 160), rng.randint(12, 127), rng.randint(1, 8))
                           for _ in range(rng.randint(2, 4)))
        return dict(kind=kind, members=members, nq=rng.randint(1, 8), split=rng.randint(1, 3))
    if kind == "lin":
        mode = rng.choice(["tl", "ad"])
        return dict(kind=kind, mode=mode, n=_log_int(rng, 24, 80), npz=rng.randint(12, 64), nq=rng.randint(1, 4),
                    hord=rng.choice([5, 8]), kord=4, split=rng.randint(1, 6))
    if kind == "fields":
        return dict(kind=kind, n=_log_int(rng, 24, 256), npz=npz, precision=rng.choice(["mixed", "mixed", "fp64"]))
    if kind == "host":
        return dict(kind=kind, n=_log_int(rng, 24, 200), npz=npz, nq=rng.randint(1, 12), split=rng.randint(1, 3))
    return dict(kind=kind, n=_log_int(rng, 20, 72), npz=npz, nq=rng.randint(1, 4), hord=rng.choice([8, 8, 5]),
                kord=rng.choice([9, 4]), split=rng.randint(1, 3))


# ------------------------------------------------------------------- inputs ---
@functools.lru_cache(maxsize=None)
def _grid(n, cube):
    """Geometry of the cube or of one face; halo cells and the cells they copy; winds of two flow directions."""
    topo = G.cube_topology()
    geoms = G.cube_geometry(n, NG) if cube else [G.tile_geometry(n, 0, NG)]
    nd = n + 2 * NG
    halo = None
    if cube:
        dst, src = [], []
        inside = range(1, n + 1)
        outside = [*range(1 - NG, 1), *range(n + 1, n + NG + 1)]
        for t in range(6):
            for j, i in [(j, i) for j in inside for i in outside] + [(j, i) for j in outside for i in inside]:
                u, si, sj = G.halo_source(topo, n, t, i, j)
                dst.append((t * nd + j + NG - 1) * nd + i + NG - 1)
                src.append((u * nd + sj + NG - 1) * nd + si + NG - 1)
        halo = (torch.tensor(dst, device=DEV), torch.tensor(src, device=DEV))
    winds = []
    for u0 in (40.0, -40.0):
        flux = []
        for g in geoms:
            psi = S.solid_body_psi(g.corners, u0) + 0.15 * abs(u0) * G.RADIUS * _waves(g.corners)
            flux.append(S.area_fluxes_from_psi(psi))
        cc = [S.courant_from_area_flux(g, ax, ay) for g, (ax, ay) in zip(geoms, flux)]
        cfl = max(max(np.abs(x[NG:-NG]).max(), np.abs(y[:, NG:-NG]).max()) for x, y in cc)
        cx = torch.tensor(np.stack([x for x, _ in cc]), device=DEV)[:, None] / cfl
        cy = torch.tensor(np.stack([y for _, y in cc]), device=DEV)[:, None] / cfl
        if cube:
            S._sync_edges(cx, cy, n, topo, row_off=NG)
            S.fill_courant_halo(cx, cy, n, NG, topo)
        winds.append((cx, cy))
    m = {k: torch.tensor(np.stack([getattr(g, k) for g in geoms]), device=DEV)
         for k in ("dx", "dy", "dxa", "dya", "area", "rarea", "centers")}
    m["sin"] = torch.tensor(np.stack([g.sin_sg[:4] for g in geoms]), device=DEV)
    return dict(geoms=geoms, topo=topo, halo=halo, winds=winds, m=m)


def _waves(p):
    x, y, z = p[..., 0], p[..., 1], p[..., 2]
    return np.sin(7 * x + 1) * np.cos(6 * y) / 7 + np.sin(9 * z) * np.cos(8 * x + 2) / 9


def _fill_halo(x, halo):
    """Edge-halo cells of (6, planes, nd, nd) from the neighbouring faces, in place."""
    dst, src = halo
    v = x.transpose(0, 1).reshape(x.shape[1], -1)
    for p in range(0, v.shape[0], 256):
        w = v[p:p + 256]
        w[:, dst] = w[:, src]
    x.copy_(v.reshape(x.shape[1], x.shape[0], *x.shape[2:]).transpose(0, 1))
    return x


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 11)
    return g


def _area_flux(gr, cx, cy, sl=slice(None)):
    """Area fluxes of (tiles, levels) Courant numbers on every row / column of the data domain."""
    m, n = gr["m"], gr["geoms"][0].n
    f = slice(NG, NG + n + 1)
    up = lambda a, s: (m[a] * m["sin"][:, s])  # noqa: E731
    xp, xn = up("dxa", 2)[:, :, NG - 1:NG + n], up("dxa", 0)[:, :, NG:NG + n + 1]
    yp, yn = up("dya", 3)[:, NG - 1:NG + n], up("dya", 1)[:, NG:NG + n + 1]
    dy, dx = m["dy"][:, :, f], m["dx"][:, f]
    return (torch.where(cx > 0, cx * (xp * dy)[:, None], cx * (xn * dy)[:, None]),
            torch.where(cy > 0, cy * (yp * dx)[:, None], cy * (yn * dx)[:, None]))


def _fields(n, npz, nq, tiles, cube, seed, smooth=False, dtype=torch.float64):
    """One step's fields: level winds of either direction (Courant numbers up to 0.8), perturbed hybrid layers with
    ps 950-1030 hPa, upwind mass fluxes, and tracers (cosine bells and Gaussians with 1 % noise, clipped at zero; or
    positive and nowhere flat)."""
    gr, g = _grid(n, cube), _gen(seed)
    rep = lambda a: a if cube else a.expand(tiles, *a.shape[1:])  # noqa: E731
    nd, f8 = n + 2 * NG, torch.float64
    rnd = lambda *s: torch.rand(*s, generator=g, device=DEV, dtype=f8)  # noqa: E731
    # a faster and a slower band of levels; the flow turns round with height
    w = 0.8 * (0.35 + 0.65 * rnd(1 if cube else tiles, npz, 1, 1))
    back = rnd(1 if cube else tiles, npz, 1, 1) < 0.3
    (ax, ay), (bx, by) = gr["winds"]
    cx = (torch.where(back, bx, ax) * w).expand(tiles, npz, nd, n + 1).contiguous()
    cy = (torch.where(back, by, ay) * w).expand(tiles, npz, n + 1, nd).contiguous()
    ak, bk = G.hybrid_levels(npz)
    dak, dbk = torch.tensor(np.diff(ak), device=DEV), torch.tensor(np.diff(bk), device=DEV)
    ref = dak[:, None, None] + dbk[:, None, None] * (95000.0 + 8000.0 * rnd(tiles, 1, nd, nd))
    dp = ref * (0.9 + 0.2 * rnd(tiles, npz, nd, nd))
    dp *= ref.sum(1, keepdim=True) / dp.sum(1, keepdim=True)
    del ref
    if cube:
        _fill_halo(dp, gr["halo"])
    s = slice(NG, NG + n)
    xf, yf = _area_flux(gr, cx, cy)
    mfx = xf[:, :, s] * torch.where(cx[:, :, s] > 0, dp[:, :, s, NG - 1:NG + n], dp[:, :, s, NG:NG + n + 1])
    mfy = yf[..., s] * torch.where(cy[..., s] > 0, dp[:, :, NG - 1:NG + n, s], dp[:, :, NG:NG + n + 1, s])
    del xf, yf
    if cube:
        S._sync_edges(mfx, mfy, n, gr["topo"], row_off=0)
    q = torch.empty(tiles, nq, npz, nd, nd, device=DEV, dtype=dtype)
    vert = 0.6 + 0.4 * torch.cos(torch.linspace(0.0, math.pi, npz, device=DEV, dtype=f8))[:, None, None]
    cen = rep(gr["m"]["centers"])
    for iq in range(nq):
        c = torch.randn(1 if cube else tiles, 1, 1, 3, generator=g, device=DEV, dtype=f8)
        if not cube:
            c = c * 0.3 + cen[:, n // 2:n // 2 + 1, n // 2:n // 2 + 1]  # on the face
        c = c / c.norm(dim=-1, keepdim=True)
        cosr = (cen * c).sum(-1)
        if iq % 2 or smooth:
            base = torch.exp(-(2 - 2 * cosr) / 0.0625)
        else:
            r = torch.arccos(cosr.clamp(-1, 1))
            base = torch.where(r < 1 / 3, 0.5 * (1 + torch.cos(3 * math.pi * r)), 0.0)
        v = base[:, None] * vert
        noise = rnd(tiles, npz, nd, nd) * 2 - 1
        v = v + 0.2 + 0.005 * noise if smooth else (v + 0.01 * noise).clamp_(min=0.0)
        if cube:
            _fill_halo(v, gr["halo"])
        q[:, iq] = v
    return dict(Q=q, DELP=dp.to(dtype), CX=cx.to(dtype), CY=cy.to(dtype), MFX=mfx.to(dtype), MFY=mfy.to(dtype)), ak, bk


# -------------------------------------------------------------- preparation ---
FIELDS = ("Q", "DELP", "CX", "CY", "MFX", "MFY")


def _state(case, cube, tiles, precision, ak, bk, **kw):
    gr = _grid(case["n"], cube)
    st = api.CubeState(case["n"], case["npz"], case["nq"], precision=precision, ntiles=tiles, **kw)
    st.set_grid(gr["geoms"] if cube else gr["geoms"] * tiles)
    st.set_levels(ak, bk)
    return st


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _upload(st, fields, names=FIELDS):
    for k in names:
        st.upload_device(k, fields[k].data_ptr(), _stream())


def _members(case):
    return [dict(kind="step", n=n, npz=k, nq=case["nq"], tiles=c, indep=True, precision="mixed", hord=8, kord=9,
                 split=case["split"], nord=0, trdm=0.0, fill=False, mass_fix=False)
            for n, k, c in (map(int, m.split("x")) for m in case["members"].split(","))]


def _make_step(case, seed):
    cube = not case["indep"] and case["tiles"] == 6
    dtype = torch.float64 if case["precision"] == "fp64" else torch.float32
    f, ak, bk = _fields(case["n"], case["npz"], case["nq"], case["tiles"], cube, seed, dtype=dtype)
    st = _state(case, cube, case["tiles"], case["precision"], ak, bk, hord=case["hord"], kord=case["kord"],
                nord_tr=case["nord"], trdm=case["trdm"], fill=case["fill"], mass_fix=case["mass_fix"],
                independent_tiles=case["indep"])
    return dict(st=st, fields=f, out=torch.empty_like(f["Q"]))


def _pin(a):
    return a.cpu().pin_memory()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        return dict(_make_step(case, seed), case=case)
    if kind == "ensemble":
        ms = [_make_step(m, seed * 31 + i) for i, m in enumerate(_members(case))]
        return dict(case=case, members=ms, ens=api.Ensemble([m["st"] for m in ms]))
    if kind == "dropin":
        f, ak, bk = _fields(case["n"], case["npz"], case["nq"], 1, False, seed)
        h = {k: np.ascontiguousarray(v[0].cpu().numpy()) for k, v in f.items()}
        # the Lagrangian interfaces at the call's end and the hybrid ones under the same surface pressure
        dp2 = _dp_end(_grid(case["n"], False), f, case["split"])[0, :, NG:-NG, NG:-NG].cpu().numpy()
        pe1 = np.concatenate([np.full((1,) + dp2.shape[1:], ak[0]), ak[0] + np.cumsum(dp2, axis=0)])
        pe2 = ak[:, None, None] + bk[:, None, None] * pe1[-1]
        return dict(case=case, host=h, work={k: v.copy() for k, v in h.items()}, pe1=pe1, pe2=pe2,
                    grid=api.GridStruct(_grid(case["n"], False)["geoms"][0]), bd=api.bounds_for(case["n"]),
                    out=np.zeros_like(h["Q"]))
    prec = case.get("precision", "fp64" if kind == "lin" else "mixed")
    dtype = torch.float64 if prec == "fp64" else torch.float32
    c = dict(case, nq=case.get("nq", 1))
    f, ak, bk = _fields(c["n"], c["npz"], c["nq"], 6, True, seed, smooth=kind == "lin", dtype=dtype)
    st = _state(c, True, 6, prec, ak, bk, hord=c.get("hord", 8), kord=c.get("kord", 9))
    s = dict(case=case, st=st, fields=f)
    if kind == "host":
        s["host"] = {k: _pin(v) for k, v in f.items()}
        s["out"] = torch.zeros_like(s["host"]["Q"]).pin_memory()
        del s["fields"]
        return s
    _upload(st, f)
    if kind == "lin":  # a perturbation relative to the trajectory
        s["pert"] = f["Q"] * torch.randn(f["Q"].shape, generator=_gen(seed + 1000), device=DEV, dtype=dtype)
        s["out"] = torch.zeros_like(f["Q"])
    else:
        st.tracer_2d(2, _stream())
        s["in"] = _field_inputs(case, seed, dtype)
        s["outs"] = {k: torch.zeros_like(v) for k, v in s["in"].items()}
    torch.cuda.synchronize()
    return s


_KINDS = {"pt": dict(kind=0, iv=1, q_min=184.0, log_p=True), "u": dict(kind=1, iv=-1), "v": dict(kind=2, iv=-1)}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        _upload(s["st"], s["fields"])
        s["st"].step(case["split"], stream=_stream())
        s["st"].download_device("Q_REMAPPED", s["out"].data_ptr(), _stream())
        return s["out"]
    if kind == "ensemble":
        for m in s["members"]:
            _upload(m["st"], m["fields"])
        s["ens"].step(case["split"], _stream())
        for m in s["members"]:
            m["st"].download_device("Q_REMAPPED", m["out"].data_ptr(), _stream())
        return [m["out"] for m in s["members"]]
    if kind == "lin":
        f = s["st"].step_tl if case["mode"] == "tl" else s["st"].step_ad
        f(case["split"], s["pert"].data_ptr(), s["out"].data_ptr(), stream=_stream())
        return s["out"]
    if kind == "fields":
        for k, a in _KINDS.items():
            s["st"].remap_fields(s["in"][k].data_ptr(), s["outs"][k].data_ptr(), 1, stream=_stream(), **a)
        return s["outs"]
    if kind == "host":
        h = s["host"]
        s["st"].step_host(case["split"], h["Q"].data_ptr(), {k: h[k].data_ptr() for k in FIELDS[1:]},
                          s["out"].data_ptr(), True)
        return s["out"]
    w, n, k = s["work"], case["n"], case["npz"]
    for f in FIELDS:  # the call updates its arguments in place
        np.copyto(w[f], s["host"][f])
    api.tracer_2d(w["Q"], w["DELP"], w["MFX"], w["MFY"], w["CX"], w["CY"], s["grid"], s["bd"], n + 1, n + 1, k,
                  case["nq"], case["hord"], case["split"], 0.0)
    api.map_scalar_3d(k, s["pe1"], w["Q"], None, k, s["pe2"], s["out"], 1, n, 1, n, 1 - NG, n + NG, 1 - NG, n + NG,
                      case["nq"], 0, case["kord"], 0.0)
    return dict(q=w["Q"][..., NG:-NG, NG:-NG], remapped=s["out"][..., NG:-NG, NG:-NG])


# --------------------------------------------------------------------- work ---
# Operations of one tracer cell: 172 in a substep (hord 8: 115 additions and multiplications, 57 min / max / signs)
# and 44 in the remap.
def _step_work(n, npz, nq, tiles, split, size):
    cells = tiles * n * n * npz
    return {"bytes": size * cells * (2 * nq + 5), "flops": cells * nq * (split * 172.0 + 44.0)}


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        w = [work(m) for m in _members(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    if kind == "fields":
        cells = 6 * case["n"] ** 2 * case["npz"]
        return {"bytes": (8 if case["precision"] == "fp64" else 4) * cells * 7, "flops": cells * 3 * 44.0}
    if kind == "lin":  # trajectory and tangent (or adjoint) of every operation
        w = _step_work(case["n"], case["npz"], case["nq"], 6, case["split"], 8)
        return {"bytes": 1.5 * w["bytes"], "flops": 3 * w["flops"]}
    size = 4 if kind == "host" or case.get("precision") == "mixed" else 8
    tiles = {"host": 6, "dropin": 1}.get(kind) or case["tiles"]
    return _step_work(case["n"], case["npz"], case["nq"], tiles, max(case["split"], 1), size)


# -------------------------------------------------------------------- exact ---
# The schemes restated in 64-bit torch: the two-dimensional flux-form transport with PPM faces (hord 8 and 5), its
# one-sided values at the edges of a face and the corner rotation, and the column remap (kord 9 and 4).
def _sgn(a, b):
    return torch.where(b < 0, -a.abs(), a.abs())


def _cw84(bl, br):
    d, t = br - bl, 3 * (br - bl) * (bl + br)
    flat = bl * br >= 0
    lo, hi = -t > d * d, t > d * d
    return (torch.where(flat, 0.0, torch.where(lo, -2 * br, bl)), torch.where(flat, 0.0, torch.where(~lo & hi, -2 * bl, br)))


def _ppm(x, c, dxa, hord):
    """Face values 1..n+1 along the last axis from cells -2..n+3 of a whole face (cell i at index i + 2)."""
    M = x.shape[-1]
    n = M - 6
    X = lambda a: x[..., a]  # noqa: E731
    lo, hi = slice(2, n + 4), slice(3, n + 5)  # cells 0..n+1, and the interface above each
    if hord == 8:
        dm = torch.zeros_like(x)
        a, b, d = x[..., :-2], x[..., 1:-1], x[..., 2:]
        xt = 0.25 * (d - a)
        mx = torch.maximum(torch.maximum(a, b), d) - b
        mn = b - torch.minimum(torch.minimum(a, b), d)
        dm[..., 1:-1] = _sgn(torch.minimum(torch.minimum(xt.abs(), mx), mn), xt)
        al = torch.zeros_like(x)
        al[..., 1:] = 0.5 * (x[..., :-1] + x[..., 1:]) + (dm[..., :-1] - dm[..., 1:]) / 3
        two = 2 * dm[..., lo]
        bl = -_sgn(torch.minimum(two.abs(), (al[..., lo] - x[..., lo]).abs()), two)
        br = _sgn(torch.minimum(two.abs(), (al[..., hi] - x[..., lo]).abs()), two)
    else:
        al = torch.zeros_like(x)
        al[..., 2:-1] = 7 / 12 * (x[..., 1:-2] + x[..., 2:-1]) - 1 / 12 * (x[..., :-3] + x[..., 3:])
        bl, br = al[..., lo] - x[..., lo], al[..., hi] - x[..., lo]
    D = lambda a: dxa[..., a]  # noqa: E731
    for e, east in ((3, False), (n + 3, True)):
        xl = ((2 * D(e - 1) + D(e - 2)) * X(e - 1) - D(e - 1) * X(e - 2)) / (D(e - 2) + D(e - 1))
        xr = ((2 * D(e) + D(e + 1)) * X(e) - D(e) * X(e + 1)) / (D(e) + D(e + 1))
        a0 = 0.5 * (xl + xr)
        o = 2  # bl, br index of cell a is a - o
        if hord == 8:
            a0 = torch.minimum(torch.maximum(a0, torch.minimum(X(e - 1), X(e))), torch.maximum(X(e - 1), X(e)))
            s11, s14, s15 = 11 / 14, 4 / 7, 3 / 14
            m = lambda a: dm[..., a]  # noqa: E731
            if not east:
                ap = s15 * X(e) + s11 * X(e + 1) - s14 * m(e + 1)
                v = {e - 1: (s14 * m(e - 2) + s11 * (X(e - 2) - X(e - 1)), a0 - X(e - 1)), e: (a0 - X(e), ap - X(e)),
                     e + 1: (ap - X(e + 1), 0.5 * (X(e + 1) + X(e + 2)) + (m(e + 1) - m(e + 2)) / 3 - X(e + 1))}
            else:
                am = s15 * X(e - 1) + s11 * X(e - 2) + s14 * m(e - 2)
                v = {e - 2: (0.5 * (X(e - 3) + X(e - 2)) + (m(e - 3) - m(e - 2)) / 3 - X(e - 2), am - X(e - 2)),
                     e - 1: (am - X(e - 1), a0 - X(e - 1)), e: (a0 - X(e), s11 * (X(e + 1) - X(e)) - s14 * m(e + 1))}
            for a, (l, r) in v.items():
                bl[..., a - o], br[..., a - o] = _cw84(l, r)
        else:
            c1, c2, c3 = -2 / 14, 11 / 14, 5 / 14
            aM = c1 * X(e - 3) + c2 * X(e - 2) + c3 * X(e - 1)
            aP = c3 * X(e) + c2 * X(e + 1) + c1 * X(e + 2)
            if e - 2 - o >= 0:
                br[..., e - 2 - o] = aM - X(e - 2)
            bl[..., e - 1 - o], br[..., e - 1 - o] = aM - X(e - 1), a0 - X(e - 1)
            bl[..., e - o], br[..., e - o] = a0 - X(e), aP - X(e)
            if e + 1 - o < bl.shape[-1]:
                bl[..., e + 1 - o] = aP - X(e + 1)
    b0, a = bl + br, c.abs()
    up, dn = slice(0, n + 1), slice(1, n + 2)
    xc = x[..., lo]
    fl = xc[..., up] + (1 - a) * (br[..., up] - a * b0[..., up])
    fr = xc[..., dn] + (1 - a) * (bl[..., dn] - a * b0[..., dn])
    if hord != 8:
        sm = bl * br < 0
        keep = sm[..., up] | sm[..., dn]
        fl, fr = torch.where(keep, fl, xc[..., up]), torch.where(keep, fr, xc[..., dn])
    return torch.where(c > 0, fl, fr)


@functools.lru_cache(maxsize=None)
def _corner_index(n, direction):
    nd, dst, src = n + 2 * NG, [], []
    out = [*range(1 - NG, 1), *range(n + 1, n + NG + 1)]
    for j in out:
        for i in out:
            su, sv = (-1 if i < 1 else 1), (-1 if j < 1 else 1)
            px, py = (1 if su < 0 else 2 * n + 1), (1 if sv < 0 else 2 * n + 1)  # twice the corner point
            u, v = 2 * i - px, 2 * j - py
            u, v = (-v, u) if (su == -sv if direction == 1 else su == sv) else (v, -u)
            dst.append((j + NG - 1) * nd + i + NG - 1)
            src.append(((v + py) // 2 + NG - 1) * nd + (u + px) // 2 + NG - 1)
    return torch.tensor(dst, device=DEV), torch.tensor(src, device=DEV)


def _corners(q, n, direction):
    dst, src = _corner_index(n, direction)
    v = q.clone().view(*q.shape[:-2], -1)
    v[..., dst] = v[..., src]
    return v.view(q.shape)


def _dp_end(gr, f, split):
    """Layer thickness after the substeps, data domain (halo as given)."""
    n = gr["geoms"][0].n
    s = slice(NG, NG + n)
    dp = f["DELP"].double().clone()
    fx, fy = f["MFX"].double(), f["MFY"].double()
    dp[..., s, s] += (fx[..., :-1] - fx[..., 1:] + fy[..., :-1, :] - fy[..., 1:, :]) * gr["m"]["rarea"][:, None, s, s]
    return dp


def _transport(gr, cube, f, q, hord, split):
    """tracer_2d of one tracer (tiles, levels, nd, nd), all tiles and levels given."""
    m, n = gr["m"], gr["geoms"][0].n
    s, r = slice(NG, NG + n), 1.0 / split
    cx, cy, mfx, mfy = (f[k].double() * r for k in ("CX", "CY", "MFX", "MFY"))
    xf, yf = _area_flux(gr, cx, cy)
    area, rarea = m["area"][:, None], m["rarea"][:, None]
    dxa, dyaT = m["dxa"][:, None], m["dya"][:, None].transpose(-1, -2)
    rax = area[..., s] + xf[..., :-1] - xf[..., 1:]
    ray = area[..., s, :] + yf[..., :-1, :] - yf[..., 1:, :]
    cyT = cy.transpose(-1, -2)
    dp, ring = f["DELP"].double().clone(), q.clone()
    for it in range(split):
        if cube:
            _fill_halo(q, gr["halo"])
        elif it:
            ring[..., s, s] = q[..., s, s]
            q = ring.clone()
        fy2 = _ppm(_corners(q, n, 2).transpose(-1, -2), cyT, dyaT, hord).transpose(-1, -2)
        qi = (q[..., s, :] * area[..., s, :] + (yf * fy2)[..., :-1, :] - (yf * fy2)[..., 1:, :]) / ray
        fx = _ppm(qi, cx[..., s, :], dxa[..., s, :], hord)
        fx2 = _ppm(_corners(q, n, 1), cx, dxa, hord)
        qj = (q[..., s] * area[..., s] + (xf * fx2)[..., :-1] - (xf * fx2)[..., 1:]) / rax
        fy = _ppm(qj.transpose(-1, -2), cyT[..., s, :], dyaT[..., s, :], hord).transpose(-1, -2)
        fx = 0.5 * (fx + fx2[..., s, :]) * mfx
        fy = 0.5 * (fy + fy2[..., s]) * mfy
        d1 = dp[..., s, s].clone()
        ra = rarea[..., s, s]
        d2 = d1 + (mfx[..., :-1] - mfx[..., 1:] + mfy[..., :-1, :] - mfy[..., 1:, :]) * ra
        new = (q[..., s, s] * d1 + (fx[..., :-1] - fx[..., 1:] + fy[..., :-1, :] - fy[..., 1:, :]) * ra) / d2
        q = q.clone()
        q[..., s, s] = new
        dp[..., s, s] = d2
    return q


def _pairwise(x):
    return torch.minimum(x[:-1], x[1:]), torch.maximum(x[:-1], x[1:])


def _remap(q, pe1, pe2, kord, iv, q_min):
    """Columns (km, cols) from interfaces pe1 onto pe2 (km + 1, cols)."""
    km = q.shape[0]
    dp = pe1[1:] - pe1[:-1]
    floor = q_min if iv == 1 else 0.0
    D = q[1:] - q[:-1]  # D[u-1] is the jump across interface u
    a = torch.empty_like(pe1)
    if kord == 9:
        g, gb = dp[1] / dp[0], dp[km - 2] / dp[km - 1]
        up, y = torch.empty_like(pe1), torch.empty_like(pe1)
        up[0], y[0] = (g + 1) / g, (g * (2 * g + 3) * q[0] + q[1]) / (g + 1) / g
        for k in range(1, km):
            d = dp[k - 1] / dp[k]
            den = 2 * (1 + d) - up[k - 1]
            up[k], y[k] = d / den, (3 * (q[k - 1] + d * q[k]) - y[k - 1]) / den
        rhs = (gb * (2 * gb + 3) * q[km - 1] + q[km - 2]) / (gb + 1)
        a[km] = (rhs - (gb + 1) * y[km - 1]) / (gb - (gb + 1) * up[km - 1])
        for k in range(km - 1, -1, -1):
            a[k] = y[k] - up[k] * a[k + 1]
        lo, hi = _pairwise(q)
        dl, dr = torch.cat([D[:1], D[:-1]]), torch.cat([D[1:], D[-1:]])
        mono = ((dl > 0) & (dr > 0)) | ((dl < 0) & (dr < 0))
        mid = a[1:km]
        below = torch.minimum(mid, hi)
        if iv >= 0:
            below = below.clamp(min=floor)
        a[1:km] = torch.where(mono, torch.minimum(torch.maximum(mid, lo), hi),
                              torch.where(dl > 0, torch.maximum(mid, lo), below))
        a[0] = torch.minimum(torch.maximum(a[0], lo[0]), hi[0])
        a[km] = torch.minimum(torch.maximum(a[km], lo[-1]), hi[-1])
        dm = None
    else:
        dm = torch.zeros_like(q)
        d0, d1, d2 = dp[:-2], dp[1:-1], dp[2:]
        dq = d1 / (d0 + d1 + d2) * ((2 * d0 + d1) / (d2 + d1) * D[1:] + (d1 + 2 * d2) / (d0 + d1) * D[:-1])
        mx = torch.maximum(torch.maximum(q[:-2], q[1:-1]), q[2:]) - q[1:-1]
        mn = q[1:-1] - torch.minimum(torch.minimum(q[:-2], q[1:-1]), q[2:])
        dm[1:-1] = _sgn(torch.minimum(torch.minimum(0.5 * dq.abs(), mx), mn), dq)
        hm, h0, h1, h2 = dp[:-3], dp[1:-2], dp[2:-1], dp[3:]
        s01, sall = h0 + h1, hm + h0 + h1 + h2
        cc = h0 / s01 + 2 * h1 * h0 / s01 * ((hm + h0) / (2 * h0 + h1) - (h2 + h1) / (2 * h1 + h0)) / sall
        c2, c3 = h0 * (hm + h0) / (2 * h0 + h1) / sall, h1 * (h1 + h2) / (h0 + 2 * h1) / sall
        a[2:km - 1] = q[1:-2] + cc * D[1:-1] - 2 * c2 * dm[2:-1] + 2 * c3 * dm[1:-2]
        for u, (k0, k1, k2) in ((1, (0, 1, 2)), (km - 1, (km - 1, km - 2, km - 3))):
            h0, h1, h2 = dp[k0], dp[k1], dp[k2]
            w0 = h1 * (h1 + h2) / ((h0 + h1) * (h0 + h1 + h2))
            w2 = -h0 * h1 / ((h0 + h1 + h2) * (h1 + h2))
            v = w0 * q[k0] + (1 - w0 - w2) * q[k1] + w2 * q[k2]
            a[u] = torch.minimum(torch.maximum(v, torch.minimum(q[k0], q[k1])), torch.maximum(q[k0], q[k1]))
        a[0], a[km] = 2 * q[0] - a[1], 2 * q[km - 1] - a[km - 1]
    bl, br = a[:-1] - q, a[1:] - q
    el, er = _cw84(bl, br)
    opp = lambda x, y: ((x > 0) & (y < 0)) | ((x < 0) & (y > 0))  # noqa: E731
    i = slice(2, km - 2)
    if kord == 9:
        Dm, D0, D1, D2 = D[0:km - 4], D[1:km - 3], D[2:km - 2], D[3:km - 1]
        flat = opp(D0, D1) & (opp(Dm, D0) | opp(D1, D2))
        b, r = bl[i], br[i]
        non = 3 * (b + r).abs() > (r - b).abs()
        z = torch.zeros_like(b)

        def bound(v, p, l):
            return torch.minimum(torch.maximum(v, torch.minimum(torch.minimum(z, p), l)), torch.maximum(torch.maximum(z, p), l))
        rc, lc = bound(r, 2 * D0, 2 * D0 - 1.5 * Dm), bound(b, -2 * D1, -2 * D1 + 1.5 * D2)
        el[i], er[i] = torch.where(flat, z, torch.where(non, lc, b)), torch.where(flat, z, torch.where(non, rc, r))
    else:
        xt = 2 * dm[i]
        el[i] = -_sgn(torch.minimum(xt.abs(), bl[i].abs()), xt)
        er[i] = _sgn(torch.minimum(xt.abs(), br[i].abs()), xt)
    bl, br = el, er
    if iv >= 0:
        s6, da = -3 * (bl + br), br - bl
        inner = -s6 > da.abs()
        low = (q + bl < floor) | (q + br < floor) | (inner & (12 * s6 * (q - floor) + s6 * s6 + 3 * da * da > 0))
        safe = torch.where(s6 == 0, 1.0, s6)
        pmin = torch.minimum(q + bl, q + br)
        pmin = torch.where(inner, torch.minimum(pmin, q + s6 / 12 + da * da / (4 * safe)), pmin)
        lam = torch.where(low, torch.where(q > floor, (q - floor) / torch.where(low, q - pmin, 1.0), 0.0), 1.0)
        bl, br = lam * bl, lam * br
    l, r, s6 = q + bl, q + br, -3 * (bl + br)
    L = (torch.searchsorted(pe1[1:km].t().contiguous(), pe2.t().contiguous(), right=True)).t().contiguous()
    X = (pe2 - pe1.gather(0, L)) / dp.gather(0, L)
    # the mean of each target layer, overlap by overlap (no difference of column masses)
    out = torch.zeros_like(q)
    t, b = L[:-1], L[1:]
    Xt, Xb = X[:-1], X[1:]
    pm = lambda k, x1, x2: (l.gather(0, k) + 0.5 * (x1 + x2) * (r.gather(0, k) - l.gather(0, k) + s6.gather(0, k))  # noqa: E731
                            - s6.gather(0, k) * (x2 * x2 + x1 * x2 + x1 * x1) / 3)
    one = torch.ones_like(q)
    mass = dp.gather(0, t) * (one - Xt) * pm(t, Xt, one)
    for j in range(1, int((b - t).max()) + 1):
        k = (t + j).clamp(max=km - 1)
        full = q.gather(0, k) * dp.gather(0, k)
        part = dp.gather(0, k) * Xb * pm(k, torch.zeros_like(Xb), Xb)
        mass += torch.where(t + j < b, full, torch.where(t + j == b, part, 0.0))
    out = torch.where(t == b, pm(t, Xt, Xb), mass / (pe2[1:] - pe2[:-1]))
    return out


def _columns(x):
    """(tiles, levels, ny, nx) -> (levels, tiles * ny * nx)."""
    return x.transpose(0, 1).reshape(x.shape[1], -1)


def _pressures(dp, ak, bk):
    """Lagrangian and hybrid interfaces (levels + 1, columns) of thicknesses (levels, columns)."""
    pe1 = torch.cat([torch.full_like(dp[:1], ak[0]), ak[0] + torch.cumsum(dp, 0)])
    to = lambda v: torch.tensor(v, device=DEV)[:, None]  # noqa: E731
    return pe1, to(ak) + to(bk) * pe1[-1:]


def _exact_step(case, seed):
    cube = not case["indep"] and case["tiles"] == 6
    dtype = torch.float64 if case["precision"] == "fp64" else torch.float32
    n, npz, nq, tiles, split = case["n"], case["npz"], case["nq"], case["tiles"], case["split"]
    f, ak, bk = _fields(n, npz, nq, tiles, cube, seed, dtype=dtype)
    gr = _grid(n, cube)
    s = slice(NG, NG + n)
    pe1, pe2 = _pressures(_columns(_dp_end(gr, f, split)[..., s, s]), ak, bk)
    out = f["Q"].double()
    for iq in range(nq):
        adv = _transport(gr, cube, f, out[:, iq].clone(), case["hord"], split)
        if cube:  # the home buffer's halo strips are those of the step's start
            _fill_halo(out[:, iq], gr["halo"])
        r = _remap(_columns(adv[..., s, s]), pe1, pe2, case["kord"], 0, 0.0)
        out[:, iq, :, s, s] = r.view(npz, tiles, n, n).transpose(0, 1)
    return out


def _field_inputs(case, seed, dtype):
    g = _gen(seed + 1000)
    shape = (6, 1, case["npz"], case["n"] + 6, case["n"] + 6)
    cos = torch.cos(torch.linspace(0, 2.5, case["npz"], device=DEV))[:, None, None]
    noise = lambda a: a * torch.randn(shape, generator=g, device=DEV, dtype=dtype)  # noqa: E731
    return dict(pt=250.0 + 60.0 * cos + noise(2.0), u=20.0 * cos + noise(5.0), v=-10.0 * cos + noise(5.0))


def _exact_fields(case, seed):
    n, npz = case["n"], case["npz"]
    dtype = torch.float64 if case["precision"] == "fp64" else torch.float32
    gr = _grid(n, True)
    f, ak, bk = _fields(n, npz, 1, 6, True, seed, dtype=dtype)
    dp = _fill_halo(_dp_end(gr, f, 2), gr["halo"])
    s, lower, upper = slice(NG, NG + n), slice(NG - 1, NG + n), slice(NG, NG + n + 1)
    out = {}
    for k, x in _field_inputs(case, seed, dtype).items():
        rows, cols = (upper if k == "u" else s), (upper if k == "v" else s)
        a = _columns(dp[..., rows, cols])
        b = a if k == "pt" else _columns(dp[..., lower, s] if k == "u" else dp[..., s, lower])
        pe1, pe2 = _pressures(0.5 * (a + b), ak, bk)
        if k == "pt":
            pe1, pe2 = pe1.log(), pe2.log()
        y = torch.zeros_like(x, dtype=torch.float64)
        r = _remap(_columns(x[:, 0][..., rows, cols].double()), pe1, pe2, 9, _KINDS[k]["iv"], _KINDS[k].get("q_min", 0.0))
        v = y[:, 0][..., rows, cols]
        v.copy_(r.view(npz, 6, *v.shape[-2:]).transpose(0, 1))
        out[k] = y
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        return [exact(m, seed * 31 + i) for i, m in enumerate(_members(case))]
    if kind == "step":
        if case["fill"] or case["mass_fix"] or case["trdm"] > 0 or case["split"] == 0:
            return None  # the damping, the filler and the fixer's dithered values are not restated here
        if case["tiles"] * case["n"] ** 2 * case["npz"] * case["nq"] > 4e8:
            return None  # too long
        return _exact_step(case, seed)
    if kind == "host":
        c = dict(case, tiles=6, indep=False, precision="mixed", hord=8, kord=9, fill=False, mass_fix=False, trdm=0.0)
        return _exact_step(c, seed)
    if kind == "dropin":
        n, k, split = case["n"], case["npz"], case["split"]
        gr = _grid(n, False)
        f, ak, bk = _fields(n, k, case["nq"], 1, False, seed)
        s = slice(NG, NG + n)
        pe1, pe2 = _pressures(_columns(_dp_end(gr, f, split)[..., s, s]), ak, bk)
        q, m = [], []
        for iq in range(case["nq"]):
            # without a halo callback the ring keeps the caller's values; the corners those of the last x sweep
            a = _transport(gr, False, f, f["Q"][:, iq].clone(), case["hord"], split)[..., s, s]
            q.append(a[0])
            m.append(_remap(_columns(a), pe1, pe2, case["kord"], 0, 0.0).view(k, n, n))
        return dict(q=torch.stack(q), remapped=torch.stack(m))
    if kind == "fields":
        return _exact_fields(case, seed)
    return None  # lin: derivatives with frozen branches
