"""The FP32 substep at the face sizes where its tiling changes (26-cell tiles): windows that hold both edges (below
29 cells), last tiles of one or two cells, which the tile before also sees the edge of, and last tiles that start 26
cells before the edge and own only part of it.  Every cell, layer thickness and reconciled edge flux against the
FP64 state (itself checked against the oracle), whose kernel is tiled differently; hord 8, whose limiter is continuous.
Tolerance: relative L2 <= 1e-5, the bound of the FP32 transport."""
import numpy as np
import pytest

from fv3atm_gb300 import api
from fv3atm_gb300 import synth as S

from ._helpers import interior, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntiles,edge_sync", [(6, False), (6, True), (1, False)])
@pytest.mark.parametrize("n", [12, 26, 28, 29, 48, 52, 53, 54, 55, 81])
def test_fp32_substep_across_tile_layouts(cuda, n, ntiles, edge_sync):
    P = S.make_problem(n, 3, 2, ntiles=ntiles, seed=n, cmax=0.8)
    out = {}
    for prec in ("mixed", "fp64"):
        st = api.CubeState(n, 3, 2, precision=prec, hord=8, ntiles=ntiles, edge_sync=edge_sync)
        try:
            st.load_problem(P)
            st.tracer_2d(2)
            out[prec] = np.asarray(st.download("Q"), np.float64), np.asarray(st.download("DELP_OUT"), np.float64)
        finally:
            st.close()
    for a, b in zip(out["mixed"], out["fp64"]):
        a, b = interior(a, n), interior(b, n)
        assert np.isfinite(a).all()
        assert rel_l2(a, b) <= 1e-5
        assert np.abs(a - b).max() <= 1e-3 * np.abs(b).max()  # no cell left out
