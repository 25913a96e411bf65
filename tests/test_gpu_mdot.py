"""The multi-dot at every column count of a group (each has its own loop), alone and after full
groups, on vectors shorter than a block, of odd length and of several blocks, against numpy.

A dot of n complex products runs at most 2 ceil(n / 256) FMAs and 40 additions one after another
(a block's threads share its elements); numpy's is no longer than that.  Twice that many roundings,
relative to the sum of the products' magnitudes."""
import ctypes as C

import numpy as np
import pytest

import picuda
from picuda import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 4999])
@pytest.mark.parametrize("nv", [2, 3, 4, 5, 6, 7, 8, 11, 13, 15])
def test_multidot_column_counts(lib_built, nv, n):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    lib, ldv = picuda.load_library(), n + 3
    g = torch.Generator(device="cuda").manual_seed(nv)
    V = torch.randn((nv, ldv), dtype=torch.complex128, device="cuda", generator=g)
    w = torch.randn(n, dtype=torch.complex128, device="cuda", generator=g)
    h = torch.full((nv,), complex(np.nan, np.nan), dtype=torch.complex128, device="cuda")
    _lib.check(lib.pi_mdot_f64_noalloc(C.c_void_p(V.data_ptr()), ldv, nv, C.c_void_p(w.data_ptr()), n,
                                       C.c_void_p(h.data_ptr()), None), "pi_mdot_f64_noalloc")
    torch.cuda.synchronize()
    Vh, wh = V.cpu().numpy()[:, :n], w.cpu().numpy()
    bound = 2 * (2 * -(-n // 256) + 40) * 2.0**-53 * (np.abs(Vh) @ np.abs(wh))
    assert (np.abs(h.cpu().numpy() - Vh.conj() @ wh) <= bound).all()
