"""ln p by table (fv3g_ln.cuh) against numpy's logarithm in extended precision: within one unit in the last place, as
CUDA's log is, over the pressures of an atmosphere and on both sides of 1 Pa, where the result passes through zero."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from fv3atm_gb300 import build as B

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "fv3g_ln.cuh"
__global__ void k(const double* p, double* out, int n) {
  __shared__ double2 tab[fv3g::LN_N];
  fv3g::ln_table(tab);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = fv3g::ln_tab(p[i], tab);
}
extern "C" int ln_of(const double* p, double* out, int n) {
  k<<<256, 256>>>(p, out, n);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def ln(cuda, tmp_path_factory):
    import torch
    d = tmp_path_factory.mktemp("ln")
    (d / "ln.cu").write_text(SOURCE)
    # the flags of the file that the table is built into
    subprocess.run([B._nvcc(), *B.ARCH, *B.FLAGS, *B.FILE_FLAGS["fv3g_remap.cu"], "-I", B.CSRC, "-shared", "-o",
                    str(d / "ln.so"), str(d / "ln.cu")], check=True)
    lib = C.CDLL(str(d / "ln.so"))

    def f(p):
        x = torch.as_tensor(p, device="cuda")
        y = torch.zeros_like(x)
        torch.cuda.synchronize()
        assert lib.ln_of(C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), C.c_int(x.numel())) == 0
        return y.cpu().numpy()
    return f


@pytest.mark.parametrize("lo,hi", [(1e3, 1.1e5), (3.0, 1e3), (1.0, 3.0), (1.0, 1.004), (0.996, 1.0), (0.1875, 1.0),
                                   (0.3, 0.4), (2.9, 3.1), (1e-3, 0.1875), (1e-300, 1e300)])
def test_within_one_ulp(ln, lo, hi):
    rng = np.random.default_rng(int(lo * 1000) % 1000)
    p = np.exp(rng.uniform(np.log(lo), np.log(hi), 400_000))
    p = np.concatenate([p[(p >= lo) & (p <= hi)], np.nextafter(lo, [0.0, np.inf]), [lo, hi, 1.0]])
    want = np.log(p.astype(np.longdouble))
    got = ln(p)
    ulp = np.spacing(np.abs(want.astype(np.float64)))
    err = np.abs(got.astype(np.longdouble) - want) / np.where(p == 1.0, 1.0, ulp)
    assert float(err.max()) <= 1.0, (float(err.max()), float(p[err.argmax()]))


def test_exceptional_pressures(ln):
    got = ln(np.array([0.0, -0.0, -1.0, np.inf, np.nan, 5e-324, 2.2e-308, 1.0]))
    assert got[0] == got[1] == -np.inf and np.isnan(got[2]) and got[3] == np.inf and np.isnan(got[4])
    assert np.allclose(got[5:], np.log(np.array([5e-324, 2.2e-308, 1.0])), rtol=1e-15, atol=0.0)
