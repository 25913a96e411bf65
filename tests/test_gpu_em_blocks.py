"""Every element-major kernel that a caller can pin, the narrow blocks among them, at widths below, at and
past a block: the same bits as the 64-wide TMA kernel of 32 rows, which the other tests hold against the
oracle; and what the tuning reports can be pinned again."""
import pytest

import picuda
from tests import models as M

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda(lib_built):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


KERNELS = [("tma", 16, 64), ("tma", 64, 64), ("tma", 32, 32), ("tma", 16, 16), ("plain", 32, 64)]


@pytest.mark.parametrize("name,make", [
    ("c2_N9", lambda: M.ensemble_c2(9)),
    ("c2_N34", lambda: M.ensemble_c2(34)),
    ("pump_N33", lambda: picuda.Models.local_pump_decay(33, down=1.0, up=0.3)),
    ("scan_N130", lambda: M.scan_model(130, 1.3, 0.2, 0.05)),
])
@pytest.mark.parametrize("ncols", [2, 16, 18, 34, 66])
def test_pinned_kernels_agree(torch_cuda, name, make, ncols):
    torch = torch_cuda
    compiled = picuda.compile(make())
    n = len(compiled.basis)
    g = torch.Generator(device="cuda").manual_seed(ncols)
    x = torch.randn((n, ncols), dtype=torch.complex64, device="cuda", generator=g)
    picuda.select_element_major_kernel(compiled, ncols, "tma", 32)
    assert picuda.element_major_tuning(compiled, ncols) == {"kernel": "tma", "rows": 32, "ms": 0.0}
    ref = picuda.apply_element_major_(torch.empty_like(x), compiled, x)
    for kernel, rows, rhs in KERNELS:
        if rows == 64 and name.startswith("pump"):
            with pytest.raises(picuda.PiArgumentError):
                picuda.select_element_major_kernel(compiled, ncols, kernel, rows, rhs=rhs)
            continue
        picuda.select_element_major_kernel(compiled, ncols, kernel, rows, rhs=rhs)
        got = picuda.element_major_tuning(compiled, ncols)
        assert (got["kernel"], got["rows"], got.get("rhs", 64)) == (kernel, rows, rhs)
        y = picuda.apply_element_major_(torch.full_like(x, float("nan")), compiled, x)
        assert torch.equal(y, ref), (kernel, rows, rhs)


def test_what_the_tuner_reports_can_be_pinned(torch_cuda):
    torch = torch_cuda
    model = M.ensemble_c2(60)
    compiled, pinned = picuda.compile(model), picuda.compile(model)
    for ncols in (16, 32, 128):
        x = torch.randn((len(compiled.basis), ncols), dtype=torch.complex64, device="cuda")
        picuda.apply_element_major_(torch.empty_like(x), compiled, x)
        found = picuda.element_major_tuning(compiled, ncols)
        picuda.select_element_major_kernel(pinned, ncols, found["kernel"], found["rows"], rhs=found.get("rhs", 64))
        assert {**picuda.element_major_tuning(pinned, ncols), "ms": 0} == {**found, "ms": 0}


def test_shapes_that_do_not_exist_are_refused(torch_cuda):
    compiled = picuda.compile(M.ensemble_c2(12))
    for rows, rhs in ((16, 32), (64, 32), (32, 16), (48, 64), (32, 8)):
        with pytest.raises(picuda.PiArgumentError):
            picuda.select_element_major_kernel(compiled, 16, "tma", rows, rhs=rhs)


@pytest.mark.parametrize("make", [lambda: M.ensemble_c2(40),
                                  lambda: picuda.Models.local_pump_decay(40, down=1.0, up=0.3)])
def test_tuner_takes_short_tiles_for_small_ensembles(torch_cuda, make):
    """At N = 40 and 32 columns tiles of 16 rows take two thirds of the time of every other kernel, more
    than timings of one launch differ by."""
    torch = torch_cuda
    compiled = picuda.compile(make())
    x = torch.randn((len(compiled.basis), 32), dtype=torch.complex64, device="cuda")
    picuda.apply_element_major_(torch.empty_like(x), compiled, x)
    found = picuda.element_major_tuning(compiled, 32)
    assert (found["kernel"], found["rows"], found.get("rhs", 64)) == ("tma", 16, 64)
