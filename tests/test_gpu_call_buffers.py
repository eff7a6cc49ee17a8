"""Call buffers from the state's pool: calls on several streams and threads, each call's buffers holding whatever
earlier calls of other shapes left in them, give bit for bit what a fresh state gives."""
import threading

import numpy as np
import pytest

from fv3atm_gb300 import api
from fv3atm_gb300 import synth as S

pytestmark = pytest.mark.gpu

N, KM = 13, 9


def _calls(st, q, f, stream):
    import torch
    out = []
    with torch.cuda.stream(stream):
        for kind in (0, 1, 2):
            o = torch.zeros_like(f)
            st.remap_fields(f.data_ptr(), o.data_ptr(), 2, kind=kind, iv=-1, kord=9, log_p=kind == 0,
                            stream=stream.cuda_stream)
            out.append(o)
    stream.synchronize()
    return [o.cpu().numpy() for o in out]


def test_pool_buffers_across_streams_threads_and_calls(cuda):
    import torch
    P = S.make_problem(N, KM, 2, seed=11, cmax=0.6)
    q = torch.as_tensor(np.asarray(P.q, dtype=np.float64), device="cuda")
    f = torch.rand((6, 2, KM, N + 6, N + 6), dtype=torch.float64, device="cuda") + 1.0
    torch.cuda.synchronize()

    def state():
        st = api.CubeState(N, KM, 2, precision="fp64", hord=8, kord=4)
        st.load_problem(P)
        return st

    def lin(st, name):
        o = torch.zeros_like(q)
        getattr(st, name)(2, q.data_ptr(), o.data_ptr())
        return o.cpu().numpy()

    want = {}
    for name in ("step_tl", "step_ad", "fields"):  # each on a state that ran nothing before
        st = state()
        want[name] = _calls(st, q, f, torch.cuda.Stream()) if name == "fields" else lin(st, name)
        st.close()
    st = state()
    try:
        for _ in range(2):
            assert np.array_equal(lin(st, "step_ad"), want["step_ad"])
            assert np.array_equal(lin(st, "step_tl"), want["step_tl"])
            got = [None] * 3
            streams = [torch.cuda.Stream() for _ in got]

            def work(i):
                got[i] = _calls(st, q, f, streams[i])

            threads = [threading.Thread(target=work, args=(i,)) for i in range(len(got))]
            for t in threads:
                t.start()
            for t in threads:
                t.join()
            for g in got:
                assert all(np.array_equal(a, b) for a, b in zip(g, want["fields"]))
    finally:
        st.close()
