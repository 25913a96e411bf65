"""Element-major batches of widths that blocks of 16 or 32 right-hand sides cover with less padding
than blocks of 64: the tuned choice (at these sizes the narrow blocks, by a factor of 1.1 to 2)
against the pinned 64-wide TMA kernel, the same bits, and against the column-batch apply."""
import pytest

import picuda
from tests import models as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coords", ["reference", "population"])
@pytest.mark.parametrize("name,make", [
    ("c2_N61", lambda: M.ensemble_c2(61)),
    ("pump_N63", lambda: picuda.Models.local_pump_decay(63, down=1.0, up=0.3)),   # larger entry planes
    ("scan_N130", lambda: M.scan_model(130, 1.3, 0.2, 0.05)),                     # 66 sectors
])
@pytest.mark.parametrize("ncols", [2, 14, 16, 18, 32, 66, 94, 96])
def test_narrow_batches(lib_built, name, make, ncols, coords):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    compiled = picuda.compile(make())
    n = len(compiled.basis)
    g = torch.Generator(device="cuda").manual_seed(ncols)
    X = torch.randn((n, ncols + 2), dtype=torch.complex64, device="cuda", generator=g)[:, :ncols]  # ld > ncols
    base = torch.full((n, ncols + 2), float("nan"), dtype=torch.complex64, device="cuda")
    picuda.apply_element_major_(base[:, :ncols], compiled, X, coords=coords)  # tunes
    Y = torch.full_like(base, float("nan"))
    picuda.apply_element_major_(Y[:, :ncols], compiled, X, coords=coords)  # the choice
    ref = torch.empty((ncols, n), dtype=torch.complex64, device="cuda")
    picuda.apply_(ref, compiled, X.t().contiguous(), precision="fp32", coords=coords)
    picuda.select_element_major_kernel(compiled, ncols, "tma", 32, coords=coords)
    Z = torch.full_like(base, float("nan"))
    picuda.apply_element_major_(Z[:, :ncols], compiled, X, coords=coords)
    torch.cuda.synchronize()
    assert torch.equal(Y[:, :ncols], Z[:, :ncols]) and torch.equal(base[:, :ncols], Z[:, :ncols])
    assert torch.isnan(Y[:, ncols:].real).all()  # nothing written past the batch
    assert (Y[:, :ncols].t() - ref).abs().max() <= 2e-6 * ref.abs().max()  # as for the other widths
