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


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("ptop", [0.0, 0.997, 1.0, 300.0])
def test_field_pressures_in_ln_p(cuda, ptop, kind):
    """Interface pressures of the cells and faces in ln p, from the two sides of 1 Pa (results beside zero) and from
    a vacuum (ln 0), against the oracle remap on numpy's logarithms.  FP64: 1e-12 as for the other field remaps."""
    import torch

    import oracle as O
    n, km = 13, 9
    P = S.make_problem(n, km, 1, seed=3, cmax=0.6)
    shift = ptop - float(P.ak[0])
    st = api.CubeState(n, km, 1, precision="fp64", kord=4)
    P.ak = np.asarray(P.ak, np.float64) + shift * (np.arange(km + 1) < km)  # the top moves, the surface stays
    rng = np.random.default_rng(kind)
    f = rng.uniform(-30.0, 30.0, (6, 1, km, n + 6, n + 6))
    try:
        st.load_problem(P)
        fin = torch.as_tensor(f, device="cuda")
        fout = torch.zeros_like(fin)
        st.remap_fields(fin.data_ptr(), fout.data_ptr(), 1, kind=kind, iv=-1, kord=4, log_p=True)
        torch.cuda.synchronize()
        got = fout.cpu().numpy()
    finally:
        st.close()
    dp = P.dp if torch.is_tensor(P.dp) else torch.as_tensor(P.dp)
    dp = dp.clone().double().cpu()
    S.fill_cube_halo(dp, n, 3, P.topo)
    dp = dp.numpy()
    for t in (0, 5):
        for j in (3, 9, n + 2):
            for i in (3, 8, n + 2):
                ib, jb = (i, j - 1) if kind == 1 else (i - 1, j) if kind == 2 else (i, j)
                col = lambda jj, ii: P.ak[0] + np.concatenate([[0.0], np.cumsum(dp[t, :, jj, ii])])
                p = 0.5 * (col(j, i) + col(jb, ib))
                p2 = P.ak + np.asarray(P.bk) * p[-1]
                with np.errstate(divide="ignore"):
                    p, p2 = np.log(p), np.log(p2)
                want = O.remap_columns(p[:, None], f[t, 0, :, j, i][:, None], p2[:, None], iv=-1, kord=4)[:, 0]
                ok = np.isfinite(want)
                assert ok.all() or ptop == 0.0
                assert rel_l2(got[t, 0, ok, j, i], want[ok]) <= 1e-12
