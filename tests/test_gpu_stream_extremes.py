"""The marching FP64 substep beside infinities and NaN in the tracer and the Courant numbers: every cell that the
update of fv_tp_2d's fluxes (the windowed kernel, FP64 minima and comparisons) leaves finite is finite and equal to it,
and the others are what that update makes them.  Tolerance: relative L2 <= 1e-12 over the finite cells, as the FP64
parity tests.  Columns per lane: one at n = 40, two at n = 58."""
import numpy as np
import pytest

from fv3atm_gb300 import api
from fv3atm_gb300 import synth as S

from ._helpers import area_fluxes, interior, ra_xy, rel_l2

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-12
VALUES = {"nan": np.nan, "minus_nan": -np.nan, "inf": np.inf, "minus_inf": -np.inf}


@pytest.fixture(scope="module", params=[40, 58])
def prob(request):
    return S.make_problem(request.param, 1, 1, seed=request.param, cmax=0.9)


def _args(P, t):
    return [np.array(a[t].numpy(), dtype=np.float64) for a in (P.q, P.dp, P.mfx, P.mfy, P.cx, P.cy)]


def _update(P, t, hord, args):
    """One substep of the tile's only tracer and level from fv_tp_2d's fluxes."""
    q, dp, mfx, mfy, cx, cy = (a[0, 0] if a.ndim == 4 else a[0] for a in args)
    g, n = P.geoms[t], P.n
    with np.errstate(all="ignore"):
        xf, yf = area_fluxes(cx, cy, g)
        rax, ray = ra_xy(xf, yf, g)
        fx, fy = np.zeros((n, n + 1)), np.zeros((n + 1, n))
        c = lambda a: np.ascontiguousarray(a)
        api.fv_tp_2d(q.copy(), c(cx), c(cy), n + 1, n + 1, hord, fx, fy, c(xf), c(yf), api.GridStruct(g),
                     api.bounds_for(n), c(rax), c(ray), mfx=c(mfx), mfy=c(mfy))
        ra = interior(g.rarea, n)
        div = lambda x, y: (x[:, :-1] - x[:, 1:]) + y[:-1] - y[1:]
        d1 = interior(dp, n)
        return (interior(q, n) * d1 + div(fx, fy) * ra) / (d1 + div(mfx, mfy) * ra)


def _substep(P, t, hord, args):
    q, dp, mfx, mfy, cx, cy = (a.copy() for a in args)
    n = P.n
    api.tracer_2d(q, dp, mfx, mfy, cx, cy, api.GridStruct(P.geoms[t]), api.bounds_for(n), n + 1, n + 1, 1, 1, hord, 1,
                  P.dt)
    return interior(q[0, 0], n)


def _places(n):
    """(row, column) of a plane with its halo: inside, beside and beyond every edge, at and beyond corners"""
    e, m = n + 2, n // 2
    return [(m, m), (m, 28), (3, m), (4, m), (e, m), (e - 1, m), (m, 3), (m, 5), (m, e), (m, e - 2), (3, 3), (e, e),
            (3, e - 1), (1, m), (m, 1), (e + 1, m), (m, e + 2), (0, 0), (e + 2, e + 3), (2, e + 1)]


def _check(P, t, hord, args, what):
    want, got = _update(P, t, hord, args), _substep(P, t, hord, args)
    assert np.array_equal(np.isnan(got), np.isnan(want)), what
    inf = np.isinf(want)
    assert np.array_equal(got[inf], want[inf]), what
    ok = np.isfinite(want)
    assert ok.sum() > 0.8 * ok.size
    assert rel_l2(got[ok], want[ok]) <= FP64_TOL, what


@pytest.mark.parametrize("hord", [8, 5, 1])
@pytest.mark.parametrize("value", sorted(VALUES))
def test_tracer_with_infinities_and_nan(cuda, prob, hord, value):
    for p in _places(prob.n):
        args = _args(prob, 1)
        args[0][0, 0][p] = VALUES[value]
        _check(prob, 1, hord, args, p)


@pytest.mark.parametrize("hord", [8, 5, 1])
@pytest.mark.parametrize("a", ["nan", "inf", "minus_inf"])
@pytest.mark.parametrize("b", ["nan", "inf", "minus_inf"])
def test_tracer_with_two_of_them_near_each_other(cuda, prob, hord, a, b):
    n = prob.n
    for off in [(0, 1), (1, 0), (0, 2), (2, 0), (1, 1), (0, 3)]:
        for p in [(n // 2, 28), (3, n // 2), (n // 2, 3), (n + 1, n // 2), (n // 2, n), (4, 4), (n // 2, 12)]:
            args = _args(prob, 1)
            q = args[0][0, 0]
            q[p] = VALUES[a]
            q[p[0] + off[0], p[1] + off[1]] = VALUES[b]
            _check(prob, 1, hord, args, (off, p))


@pytest.mark.parametrize("hord", [8, 5, 1])
def test_courant_numbers_with_nan(cuda, prob, hord):
    for p in [(10, 11), (3, 0), (20, 20), (0, 4), (prob.n + 5, 9)]:
        args = _args(prob, 1)
        args[4][0][p] = np.nan
        args[5][0][p[1], p[0]] = np.nan
        _check(prob, 1, hord, args, p)
