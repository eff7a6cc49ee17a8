"""The FP32 warp-per-column remap against the FP64 oracle remap of the same advected field, at the level counts
where the levels a lane holds change (2, 3, 4 and 5 of them), with odd and single tracer counts (the second field of
a pass repeats the first) and a column count that leaves the last block partly empty.  Tolerance: relative L2 <= 2e-6
per tracer (FP32 storage of the result and of the interface solve), as for the thread-per-column form."""
import numpy as np
import pytest

from fv3atm_gb300 import api
from fv3atm_gb300 import synth as S

from ._helpers import interior, rel_l2, remap_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kord", [4, 9])
@pytest.mark.parametrize("npz,nq", [(3, 1), (31, 2), (32, 3), (63, 1), (64, 5), (95, 2), (96, 1), (127, 3), (128, 4)])
def test_warp_remap_at_the_edges_of_its_level_counts(cuda, npz, nq, kord):
    n = 13
    P = S.make_problem(n, npz, nq, seed=npz, cmax=0.8)
    st = api.CubeState(n, npz, nq, precision="mixed", kord=kord)
    try:
        st.load_problem(P)
        st.tracer_2d(2)
        q_adv, dp = st.download("Q"), st.download("DELP_OUT")
        st.remap()
        q2 = st.download("Q_REMAPPED")
    finally:
        st.close()
    ref, _, _, _ = remap_reference(q_adv, dp, P.ak, P.bk, n, kord=kord, iv=0)
    for iq in range(nq):
        a, r = interior(q2[:, iq], n), interior(ref[:, iq], n)
        assert np.isfinite(a).all()
        assert rel_l2(a, r) <= 2e-6, (iq, rel_l2(a, r))
