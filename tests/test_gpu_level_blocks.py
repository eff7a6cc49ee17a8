"""The FP64 substep where device memory does not leave room for the work planes of all levels: it goes through the
levels in blocks, with the same results bit for bit.  Another allocation holds the memory while the state is created
(or the host-array call runs); a gigabyte or more stays free."""
import threading

import numpy as np
import pytest

from fv3atm_gb300 import api
from fv3atm_gb300 import synth as S

pytestmark = pytest.mark.gpu

MIB = 1 << 20
N, KM = 96, 127


def _free():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def _hold(leave):
    import torch
    return torch.empty(max(_free() - leave, 0), dtype=torch.uint8, device="cuda")


@pytest.fixture(scope="module")
def prob():
    return S.make_problem(N, KM, 1, seed=6, cmax=0.8)


@pytest.mark.parametrize("kw", [dict(), dict(edge_sync=True, trdm=0.05, nord_tr=1, hord=5)])
def test_state_created_short_of_memory(cuda, prob, kw):
    import torch
    field = 8 * 6 * KM * 104 * 103  # bytes of a per-level field
    base = 17 * field               # the state without the work planes (8 such fields)
    out = []
    for short in (False, True):
        api.release_call_buffers()
        hold = _hold(base + 20 * field) if short else None
        before = _free()
        st = api.CubeState(N, KM, 1, precision="fp64", kord=4, **kw)
        size = before - _free()
        del hold
        torch.cuda.empty_cache()
        try:
            st.load_problem(prob)
            got = []
            for qs in (1, 3):
                st.upload("Q", prob.q.numpy())
                st.tracer_2d(qs)
                got += [st.download("Q"), st.download("DELP_OUT")]
            st.upload("Q", prob.q.numpy())
            st.step(2)
            got.append(st.download("Q_REMAPPED"))
            if not kw:
                x = torch.as_tensor(prob.q.numpy(), device="cuda")
                y = torch.zeros_like(x)
                st.step_tl(2, x.data_ptr(), y.data_ptr())
                got.append(y.cpu().numpy())
                pin = {k: torch.as_tensor(v).contiguous().pin_memory() for k, v in
                       (("Q", prob.q), ("DELP", prob.dp), ("CX", prob.cx), ("CY", prob.cy), ("MFX", prob.mfx),
                        ("MFY", prob.mfy))}
                o = torch.zeros_like(pin["Q"]).pin_memory()
                st.step_host(2, pin["Q"].data_ptr(), {k: h.data_ptr() for k, h in pin.items()}, o.data_ptr(), False)
                got.append(o.numpy().copy())
            assert st.error_code() == 0
        finally:
            st.close()
        out.append((size, got))
    assert out[1][0] < out[0][0] - 2 * field  # fewer levels held
    for a, b in zip(out[0][1], out[1][1]):
        assert np.array_equal(a, b)


def test_host_arrays_short_of_memory(cuda):
    """tracer_2d on host arrays, from threads of their own (which keep their device memory)."""
    n, km = 384, 40
    P = S.make_problem(n, km, 1, seed=8, cmax=0.8, ntiles=1)
    need = 8 * 392 * 391 * km * 11
    out = []

    def run(short):
        q, dp, mfx, mfy, cx, cy = (np.ascontiguousarray(a[0].numpy()).copy() for a in (P.q, P.dp, P.mfx, P.mfy, P.cx, P.cy))
        hold = _hold(need + 800 * MIB) if short else None
        before = _free()
        api.tracer_2d(q, dp, mfx, mfy, cx, cy, api.GridStruct(P.geoms[0]), api.bounds_for(n), n + 1, n + 1, km, 1, 8, 2, P.dt)
        out.append((before - _free(), q, dp))
        del hold
        _free()

    for short in (False, True):
        t = threading.Thread(target=run, args=(short,))
        t.start()
        t.join()
    assert len(out) == 2
    assert out[1][0] < out[0][0] - 100 * MIB
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.array_equal(a, b)
