"""The FP64 column remap where a column holds more than ordinary numbers: source layers and targets without
thickness, infinities and NaN in the field, NaN in the surface value and the target pressures.  The batched kernel's results are
finite where the general form of the schemes (the remap on caller-owned device arrays, one thread a column) has
finite ones, equal to it there, and the other columns of the call are as without them.  Tolerance: relative L2 <=
1e-12 over the finite values, as the FP64 parity tests."""
import ctypes as C

import numpy as np
import pytest

from fv3atm_gb300 import _lib, api

from ._helpers import rel_l2

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-12
NCOL = 21


def _general(pe1, q, pe2, iv, kord, q_min, qs):
    """fv3g_remap_columns_noalloc"""
    import torch
    km, kn, nfield = q.shape[1], pe2.shape[0] - 1, q.shape[0]
    d = [torch.as_tensor(np.ascontiguousarray(x), device="cuda") for x in (pe1, q, pe2)]
    s = None if qs is None else torch.as_tensor(qs, device="cuda")
    out = torch.zeros((nfield, kn, NCOL), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    p = lambda t: None if t is None else C.c_void_p(t.data_ptr())
    _lib.call("fv3g_remap_columns_noalloc", NCOL, km, p(d[0]), p(d[1]), p(s), kn, p(d[2]), p(out), nfield, iv, kord,
              C.c_double(q_min), None)
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _batched(pe1, q, pe2, iv, kord, q_min, qs):
    km, kn, nfield = q.shape[1], pe2.shape[0] - 1, q.shape[0]
    out = np.zeros((nfield, kn, 1, NCOL))
    api.map_scalar_3d(km, np.ascontiguousarray(pe1[:, None]), np.ascontiguousarray(q[:, :, None]),
                      None if qs is None else np.ascontiguousarray(qs[None]), kn, np.ascontiguousarray(pe2[:, None]),
                      out, 1, NCOL, 1, 1, 1, NCOL, 1, 1, nfield, iv, kord, q_min)
    return out[:, :, 0]


def _put(where, value):
    """value into every other column's layer (or interface) at `where` of its height"""
    def f(pe1, pe2, q, qs):
        a = {"q": q, "pe2": pe2}[where[0]]
        k = int(where[1] * (a.shape[-2] - 1))
        a[..., k, ::2] = value
    return f


def _no_thickness(where, interface):
    def f(pe1, pe2, q, qs):
        a = pe1 if where == "pe1" else pe2
        k = 1 + int(interface * (a.shape[0] - 2))
        a[k - 1 if k == a.shape[0] - 1 else k, ::2] = a[k if k == a.shape[0] - 1 else k - 1, ::2]
    return f


def _surface(pe1, pe2, q, qs):
    if qs is not None:
        qs[::2] = np.nan


EXTREMES = {
    "no_top_layer": _no_thickness("pe1", 0.0), "no_middle_layer": _no_thickness("pe1", 0.5),
    "no_bottom_layer": _no_thickness("pe1", 1.0), "no_middle_target": _no_thickness("pe2", 0.5),
    "no_bottom_target": _no_thickness("pe2", 1.0), "surface": _surface,
    **{f"{name}_{at}": _put(("q", at), v) for at in (0.0, 0.4, 1.0)
       for name, v in (("nan", np.nan), ("minus_nan", -np.nan), ("inf", np.inf), ("minus_inf", -np.inf))},
    "nan_pe2": _put(("pe2", 0.6), np.nan),
}


@pytest.mark.parametrize("extreme", sorted(EXTREMES))
@pytest.mark.parametrize("kord", [9, 4])
@pytest.mark.parametrize("km,kn", [(3, 4), (8, 8), (33, 20), (64, 64), (127, 127)])
def test_batched_remap_is_the_general_form_at_extremes(cuda, km, kn, kord, extreme):
    rng = np.random.default_rng(1000 * km + kn)
    pe1 = np.cumsum(np.vstack([np.full((1, NCOL), 100.0), rng.uniform(0.2, 2.0, (km, NCOL))]), axis=0)
    frac = np.sort(np.vstack([np.zeros((1, NCOL)), rng.uniform(size=(kn - 1, NCOL)), np.ones((1, NCOL))]), axis=0)
    pe2 = pe1[:1] + frac * (pe1[-1:] - pe1[:1])
    pe2[-1] = pe1[-1]
    q = rng.uniform(-1.0, 1.0, (3, km, NCOL))
    for iv in (-2, -1, 0, 1):
        qs = rng.uniform(size=NCOL) if iv == -2 else None
        q_min = 0.1 if iv == 1 else 0.0
        plain = _batched(pe1, q, pe2, iv, kord, q_min, qs)
        a, b, c, s = pe1.copy(), pe2.copy(), q.copy(), None if qs is None else qs.copy()
        target = c[:2]  # the last field stays as it is
        EXTREMES[extreme](a, b, target, s)
        want, got = _general(a, c, b, iv, kord, q_min, s), _batched(a, c, b, iv, kord, q_min, s)
        assert np.array_equal(np.isnan(got), np.isnan(want))
        assert np.array_equal(got[np.isinf(want)], want[np.isinf(want)])
        ok = np.isfinite(want)
        assert rel_l2(got[ok], want[ok]) <= FP64_TOL
        assert np.array_equal(got[..., 1::2], plain[..., 1::2])  # the columns without


@pytest.mark.parametrize("kord", [9, 4])
def test_more_fields_than_a_launch_takes(cuda, kord):
    """1024 fields are a launch; fields of the first, of the last of it and of the next one hold a NaN."""
    rng = np.random.default_rng(kord)
    km, nf = 5, 1030
    pe1 = np.cumsum(np.vstack([np.full((1, NCOL), 10.0), rng.uniform(0.2, 2.0, (km, NCOL))]), axis=0)
    pe2 = pe1[:1] + np.linspace(0.0, 1.0, km + 1)[:, None] * (pe1[-1:] - pe1[:1])
    pe2[-1] = pe1[-1]
    q = rng.uniform(-1.0, 1.0, (nf, km, NCOL))
    q[[0, 31, 32, 1023, 1024, 1029], 2, 3] = np.nan
    want, got = _general(pe1, q, pe2, 0, kord, 0.0, None), _batched(pe1, q, pe2, 0, kord, 0.0, None)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = np.isfinite(want)
    assert rel_l2(got[ok], want[ok]) <= FP64_TOL
