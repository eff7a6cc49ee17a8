"""CTA widths of FP64 states: the marching substep has one kind of CTA, so the autotuner picks one width and both are
reported as it (a second, for edge-ring CTAs that do not exist, used to be whichever timing noise preferred)."""
import pytest

from fv3atm_gb300 import api
from fv3atm_gb300 import synth as S
from fv3atm_gb300._lib import Fv3gError

pytestmark = pytest.mark.gpu


def test_fp64_autotune_picks_one_width(cuda):
    P = S.make_problem(24, 3, 7, seed=1, cmax=0.5)  # (wider CTAs than tracers are cut to them: 7 > 6 is refused)
    for _ in range(8):
        st = api.CubeState(24, 3, 7, precision="fp64")
        try:
            st.load_problem(P)
            w = st.autotune()
            assert st.widths() == (w, w) and 4 <= w <= 6
            st.tracer_2d(1)
        finally:
            st.close()


@pytest.mark.parametrize("warps", [1, 6, 7])
def test_fp64_widths_accepted(cuda, warps):
    P = S.make_problem(24, 3, 7, seed=1, cmax=0.5)
    st = api.CubeState(24, 3, 7, precision="fp64", warps_per_cta=warps)
    try:
        st.load_problem(P)
        if warps > 6:
            with pytest.raises(Fv3gError, match="1..6"):
                st.tracer_2d(1)
        else:
            st.tracer_2d(1)
            assert st.widths() == (warps, warps)
    finally:
        st.close()
