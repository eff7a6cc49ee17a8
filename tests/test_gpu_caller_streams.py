"""Work that a caller queues on streams of its own, one after another, acts on a state in the order of the calls: each
entry waits for what was queued on the state before it.  The earlier call is held back on its stream by a bounded spin,
so that an entry that does not wait reads (or overwrites) the field too early; results are those of the same calls on
one stream, bit for bit."""
import numpy as np
import pytest

from fv3atm_gb300 import api
from fv3atm_gb300 import synth as S

pytestmark = pytest.mark.gpu

N, KM, NQ = 30, 17, 2
SPIN = 20_000_000  # some 10 ms


def _device(x, dtype):
    import torch
    return torch.as_tensor(x).to(dtype).cuda().contiguous()


def _held(st, call):
    """call on a stream held back by a spin; a second stream for what follows"""
    import torch
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        torch.cuda._sleep(SPIN)
    call(a.cuda_stream)
    return b


@pytest.mark.parametrize("entry", ["step_tl", "step_ad"])
def test_linearised_step_after_a_held_upload(cuda, entry):
    """The step is about the field whose upload was queued before it."""
    import torch
    P = S.make_problem(N, 3, 1, seed=3, cmax=0.7)
    q = np.array(P.q.numpy())
    new = _device(0.25 + q[:, :, ::-1].copy(), torch.float64)
    x = _device(np.random.default_rng(0).standard_normal(q.shape), torch.float64)
    st = api.CubeState(N, 3, 1, precision="fp64", hord=8, kord=4)
    try:
        st.load_problem(P)
        st.upload_device("Q", new.data_ptr())
        want, got = torch.zeros_like(x), torch.zeros_like(x)
        getattr(st, entry)(2, x.data_ptr(), want.data_ptr())
        st.upload("Q", q)
        torch.cuda.synchronize()
        b = _held(st, lambda s: st.upload_device("Q", new.data_ptr(), stream=s))
        getattr(st, entry)(2, x.data_ptr(), got.data_ptr(), stream=b.cuda_stream)
        torch.cuda.synchronize()
        assert torch.equal(got, want)
    finally:
        st.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("kind", [0, 1])
def test_field_remap_after_a_held_transport(cuda, kind, precision):
    """The remap is from the thicknesses of the tracer_2d queued before it."""
    import torch
    dt = torch.float64 if precision == "fp64" else torch.float32
    P = S.make_problem(N, KM, 1, seed=5, cmax=0.9)
    f = _device(np.random.default_rng(1).uniform(1.0, 2.0, (6, 1, KM, N + 6, N + 6)), dt)
    out = []
    for held in (False, True):
        st = api.CubeState(N, KM, 1, precision=precision, kord=4)
        try:
            st.load_problem(P)
            o = torch.zeros_like(f)
            torch.cuda.synchronize()
            s = None
            if held:
                s = _held(st, lambda s: st.tracer_2d(3, stream=s)).cuda_stream
            else:
                st.tracer_2d(3)
            st.remap_fields(f.data_ptr(), o.data_ptr(), 1, kind=kind, iv=-1, kord=4, stream=s)
            torch.cuda.synchronize()
            out.append(o)
        finally:
            st.close()
    assert torch.equal(out[0], out[1])


def test_host_step_after_a_held_download(cuda):
    """A host-array step on another stream does not overwrite the field that a download queued before it still
    reads, and a later upload on the state's stream waits for the step's own downloads."""
    import torch
    P = S.make_problem(N, KM, NQ, seed=7, cmax=0.8)
    pinned = lambda a: torch.as_tensor(a).double().contiguous().pin_memory()
    host = {k: pinned(v) for k, v in (("DELP", P.dp), ("CX", P.cx), ("CY", P.cy), ("MFX", P.mfx), ("MFY", P.mfy))}
    q = pinned(P.q)
    other = _device(np.array(P.q.numpy()) * 0.5 + 0.125, torch.float64)
    st = api.CubeState(N, KM, NQ, precision="fp64")
    try:
        st.load_problem(P)
        want, got = torch.zeros_like(q).pin_memory(), torch.zeros_like(q).pin_memory()
        args = lambda o: (2, q.data_ptr(), {k: h.data_ptr() for k, h in host.items()}, o.data_ptr(), False)
        st.step_host(*args(want))
        st.upload_device("Q", other.data_ptr())
        read = torch.zeros_like(other)
        torch.cuda.synchronize()
        b = _held(st, lambda s: st.download_device("Q", read.data_ptr(), stream=s))
        st.step_host(*args(got), stream=b.cuda_stream)
        st.upload_device("Q", other.data_ptr())
        after = st.download("Q")
        torch.cuda.synchronize()
        assert torch.equal(read, other)
        assert torch.equal(got, want)
        assert np.array_equal(after, other.cpu().numpy())
    finally:
        st.close()
