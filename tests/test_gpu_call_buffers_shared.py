"""Idle call buffers of the linearised steps and field remaps are held once per device, not per state, and given back:
by release_call_buffers, and with the last state that used them."""
import numpy as np
import pytest

from fv3atm_gb300 import api
from fv3atm_gb300 import synth as S

pytestmark = pytest.mark.gpu

MIB = 1 << 20
N, KM, NQ = 64, 32, 2


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _state(P):
    st = api.CubeState(N, KM, NQ, precision="fp64", hord=5, kord=4)
    st.load_problem(P)
    return st


def test_states_share_idle_buffers_and_give_them_back(cuda):
    import torch
    P = S.make_problem(N, KM, NQ, seed=2, cmax=0.6)
    x = torch.as_tensor(np.random.default_rng(0).standard_normal(tuple(P.q.shape)), device="cuda")
    y = torch.zeros_like(x)
    call = lambda st: st.step_tl(2, x.data_ptr(), y.data_ptr())
    plane = 8 * 6 * KM * (N + 7) * (N + 7)  # bytes of a per-level field, less the rows' padding
    least = 20 * NQ * plane                 # the four sets of six weights of every face alone are 24 such fields a tracer
    first = _state(P)
    call(first)
    api.release_call_buffers()
    base = _free()  # kernels loaded, nothing idle
    call(first)
    want, one = y.clone(), _free()
    assert base - one >= least
    others = [_state(P) for _ in range(2)]
    before = _free()
    for st in others:
        call(st)
        assert torch.equal(y, want)
    assert before - _free() < 32 * MIB
    api.release_call_buffers()
    assert _free() - before >= least
    call(others[0])
    assert torch.equal(y, want)
    for st in others:
        st.close()
    held = _free()
    first.close()
    assert _free() - held >= least  # with the last state
    api.release_call_buffers()      # nothing to give back
    st = _state(P)
    call(st)
    assert torch.equal(y, want)
    st.close()
