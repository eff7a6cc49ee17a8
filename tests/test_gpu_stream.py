"""The marching FP64 substep at the edges of its strips (26, 56 and 58 output columns), its chunks along j and its
tracer groups, against the FP64 oracle."""
import numpy as np
import pytest

import oracle as O
from fv3atm_gb300 import api
from fv3atm_gb300 import synth as S

from ._helpers import interior, rel_l2

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-12  # relative L2, as the FP64 parity tests


@pytest.mark.parametrize("hord", [8, 5, 1])
@pytest.mark.parametrize("n,nq,npz", [(12, 1, 2), (26, 5, 2), (27, 2, 2), (56, 3, 3), (57, 7, 2), (58, 1, 2), (59, 9, 2),
                                      (117, 2, 2)])
def test_marching_substep_matches_oracle(cuda, n, nq, npz, hord):
    P = S.make_problem(n, npz, nq, seed=n + nq, cmax=0.9)
    ref, _, _ = O.tracer_2d_cube(P.q, P.dp, P.mfx, P.mfy, P.cx, P.cy, P.geoms, P.topo, hord=hord, q_split=2)
    st = api.CubeState(n, npz, nq, precision="fp64", hord=hord)
    st.load_problem(P)
    st.tracer_2d(2)
    got = st.download("Q")
    assert rel_l2(interior(got, n), interior(np.asarray(ref), n)) <= FP64_TOL
    assert st.error_code() == 0
    st.close()


@pytest.mark.parametrize("warps", [1, 2, 3, 6])
def test_tracer_groups_do_not_change_results(cuda, warps):
    """Groups of any size (a last one with fewer tracers included) advance every tracer alike."""
    P = S.make_problem(33, 3, 7, seed=3, cmax=0.8)
    got = []
    for w in (0, warps):
        st = api.CubeState(33, 3, 7, precision="fp64", hord=8, warps_per_cta=w)
        st.load_problem(P)
        st.tracer_2d(2)
        got.append(st.download("Q"))
        st.close()
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("kord", [9, 4])
@pytest.mark.parametrize("km,kn", [(1, 3), (2, 2), (3, 5), (4, 4), (31, 31), (32, 32), (63, 64), (64, 63), (95, 95), (96, 40),
                                   (127, 127), (128, 128), (20, 100)])
@pytest.mark.parametrize("iv", [0, 1, -1])
def test_fp64_remap_matches_oracle(cuda, km, kn, kord, iv):
    """The FP64 column remap at the level counts where its lanes' layers change, onto finer and coarser targets;
    tracers with zeros and jumps (the positivity scaling), columns that straddle several source layers."""
    rng = np.random.default_rng(100 * km + kn + kord)
    ncol = 37
    pe1 = np.cumsum(np.vstack([np.full((1, ncol), 100.0), rng.uniform(0.2, 2.0, (km, ncol))]), axis=0)
    frac = np.sort(np.vstack([np.zeros((1, ncol)), rng.uniform(0.0, 1.0, (kn - 1, ncol)), np.ones((1, ncol))]), axis=0)
    pe2 = pe1[:1] + frac * (pe1[-1:] - pe1[:1])
    pe2[-1] = pe1[-1]
    q = rng.uniform(-1.0, 1.0, (2, km, ncol))
    q[0] = np.maximum(q[0], 0.0)
    ref = np.stack([O.remap_columns(pe1, x, pe2, iv=iv, kord=kord, q_min=0.1 if iv == 1 else 0.0) for x in q])
    got = np.zeros((2, kn, 1, ncol))
    api.map_scalar_3d(km, np.ascontiguousarray(pe1[:, None]), np.ascontiguousarray(q[:, :, None]), None, kn,
                      np.ascontiguousarray(pe2[:, None]), got, 1, ncol, 1, 1, 1, ncol, 1, 1, 2, iv, kord,
                      0.1 if iv == 1 else 0.0)
    ok = np.isfinite(ref)  # kord 9's interface system of two layers is singular: the oracle divides by zero there
    assert ok.all() or (km == 2 and kord == 9)
    assert rel_l2(got[:, :, 0][ok], ref[ok]) <= FP64_TOL
