"""The linearised step about a trajectory with an infinity or a NaN: its tangent and its adjoint are NaN at the cell,
as the forward-mode derivatives there are, and those of columns and cells out of its reach are bit for bit the ones
without it; the column remap's tangent is NaN where that of the drop-in (dual numbers) is."""
import numpy as np
import pytest

from fv3atm_gb300 import api
from fv3atm_gb300 import synth as S

from ._helpers import interior, rel_l2

pytestmark = pytest.mark.gpu

N, KM = 29, 9
T, K, J, I = 2, 4, 14, 12  # tile, level, row and column (1-based) of the cell


def _state(P, hord):
    st = api.CubeState(N, KM, 1, precision="fp64", hord=hord, kord=4, iv=0)
    st.load_problem(P)
    return st


def _lin(st, name, x, parts):
    import torch
    d = torch.as_tensor(x, device="cuda")
    out = torch.zeros_like(d)
    getattr(st, name)(1, d.data_ptr(), out.data_ptr(), parts=parts)
    return interior(out.cpu().numpy(), N)[:, 0]


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("hord", [8, 5, 1])
def test_transport_about_a_nan(cuda, hord, value):
    P = S.make_problem(N, KM, 1, seed=4, cmax=0.7)
    q = np.array(P.q.numpy(), dtype=np.float64)
    x = np.random.default_rng(1).standard_normal(q.shape)
    st = _state(P, hord)
    try:
        for name in ("step_tl", "step_ad"):
            st.upload("Q", q)
            plain = _lin(st, name, x, 1)
            odd = q.copy()
            odd[T, 0, K, J + 2, I + 2] = value
            st.upload("Q", odd)
            got = _lin(st, name, x, 1)
            if hord == 8:  # (a cell beside a NaN falls to the first-order flux with the 2-dx filters)
                assert np.isnan(got[T, K, J - 1, I - 1])
            far = np.ones(got.shape, bool)
            far[T, K, J - 8:J + 7, I - 8:I + 7] = False
            assert np.array_equal(got[far], plain[far])
    finally:
        st.close()


@pytest.mark.parametrize("value", [np.nan, -np.nan, np.inf])
@pytest.mark.parametrize("level", [0, 1, 2, 4, KM - 1])
def test_column_remap_about_a_nan(cuda, level, value):
    P = S.make_problem(N, KM, 1, seed=4)
    host = lambda a: np.array(a.detach().cpu().numpy() if hasattr(a, "detach") else a, dtype=np.float64)
    q, delp = host(P.q), host(P.dp)
    x = np.random.default_rng(2).standard_normal(q.shape)
    st = _state(P, 8)
    try:
        st.upload("Q", q)
        plain, plain_ad = _lin(st, "step_tl", x, 2), _lin(st, "step_ad", x, 2)
        q[T, 0, level, 3:3 + N:2, 3:3 + N] = value
        st.upload("Q", q)
        got, got_ad = _lin(st, "step_tl", x, 2), _lin(st, "step_ad", x, 2)
    finally:
        st.close()
    clean = np.ones((N, N), bool)
    clean[::2] = False
    for a, b in ((got, plain), (got_ad, plain_ad)):
        assert np.array_equal(a[T][:, clean], b[T][:, clean])
        assert np.array_equal(a[[0, 1, 3, 4, 5]], b[[0, 1, 3, 4, 5]])
    c = slice(3, 3 + N)
    row = lambda a: np.ascontiguousarray(a[:, c, c].reshape(a.shape[0], 1, N * N))
    d = row(delp[T])[:, 0]
    pe1 = np.concatenate([np.full((1, N * N), P.ak[0]), P.ak[0] + np.cumsum(d, axis=0)])
    pe2 = np.asarray(P.ak)[:, None] + np.asarray(P.bk)[:, None] * pe1[-1]
    want = np.zeros((KM, 1, N * N))
    api.map1_ppm_tl(KM, np.ascontiguousarray(pe1), row(q[T, 0]), row(x[T, 0]), None, KM, np.ascontiguousarray(pe2), None,
                    want, 1, N * N, 1, 1, N * N, 1, 1, 0, 4)
    want = want.reshape(KM, N, N)
    assert np.array_equal(np.isnan(got[T]), np.isnan(want))
    ok = np.isfinite(want)
    assert rel_l2(got[T][ok], want[ok]) <= 1e-12
