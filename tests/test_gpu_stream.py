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
