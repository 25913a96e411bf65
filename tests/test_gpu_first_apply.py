"""The first apply of a plan, which lays out its coefficient planes, beside other work on the plan."""
import threading
import time

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


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_first_apply_does_not_wait_for_a_running_solve(torch_cuda, precision):
    """Mixed RK4 keeps the plan's own stream busy for a good part of a second and lays out no planes of
    either precision; meanwhile the first apply on another stream comes back in a small part of that."""
    torch = torch_cuda
    model = M.ensemble_c2(120)
    dtype = torch.complex128 if precision == "fp64" else torch.complex64
    n = len(model.basis)
    x = torch.randn(n, dtype=dtype, device="cuda")
    y, ref = torch.zeros_like(x), torch.zeros_like(x)
    rho = torch.from_numpy(picuda.computational_product_state(model.basis, 2).data).cuda()
    warm = picuda.compile(model)  # loads the kernels
    picuda.apply_(ref, warm, x, precision=precision)
    picuda.evolve_(torch.empty_like(rho), warm, rho, (0.0, 1e-3), steps=8, precision="mixed")
    torch.cuda.synchronize()
    compiled = picuda.compile(model)
    span = {}
    started = threading.Event()

    def solve():
        torch.cuda.set_device(0)
        with torch.cuda.stream(torch.cuda.Stream()):
            dest = torch.empty_like(rho)
            started.set()
            span["begin"] = time.perf_counter()
            picuda.evolve_(dest, compiled, rho, (0.0, 2.5), steps=30000, precision="mixed")
            torch.cuda.current_stream().synchronize()
            span["end"] = time.perf_counter()

    t = threading.Thread(target=solve)
    t.start()
    started.wait()
    time.sleep(0.1)  # its launches are on their way
    with torch.cuda.stream(torch.cuda.Stream()):
        t0 = time.perf_counter()
        picuda.apply_(y, compiled, x, precision=precision)
        torch.cuda.current_stream().synchronize()
        took = time.perf_counter() - t0
        began_inside = "end" not in span
    t.join()
    total = span["end"] - span["begin"]
    assert began_inside and total > 0.3  # there was something to wait for
    assert took < 0.15 * total, (took, total)
    assert torch.equal(y, ref)


def test_first_applies_of_several_streams(torch_cuda):
    """Several streams that meet a new plan at once all read filled planes."""
    torch = torch_cuda
    model = M.ensemble_c2(90)
    x = torch.randn((4, len(model.basis)), dtype=torch.complex128, device="cuda")
    ref = picuda.apply_(torch.empty_like(x), picuda.compile(model), x)
    streams = [torch.cuda.Stream() for _ in range(4)]
    for _ in range(10):
        compiled = picuda.compile(model)
        ys = [torch.full_like(x, float("nan")) for _ in streams]
        torch.cuda.synchronize()
        for s, y in zip(streams, ys):
            with torch.cuda.stream(s):
                picuda.apply_(y, compiled, x)
        torch.cuda.synchronize()
        assert all(torch.equal(y, ref) for y in ys)


def test_first_element_major_apply_does_not_wait_for_a_running_solve(torch_cuda):
    """The element-major tables are filled beside the plan's own stream as well, and FP64 applies do not
    queue behind their lock."""
    torch = torch_cuda
    model = M.ensemble_c2(120)
    n = len(model.basis)
    X = torch.randn((n, 16), dtype=torch.complex64, device="cuda")
    Y, ref = torch.zeros_like(X), torch.zeros_like(X)
    rho = torch.from_numpy(picuda.computational_product_state(model.basis, 2).data).cuda()
    warm = picuda.compile(model)  # loads the kernels
    picuda.select_element_major_kernel(warm, 16, "tma", 32)
    picuda.apply_element_major_(ref, warm, X)
    dest = torch.empty_like(rho)
    picuda.evolve_(dest, warm, rho, (0.0, 1e-3), steps=8)
    torch.cuda.synchronize()
    compiled = picuda.compile(model)
    picuda.select_element_major_kernel(compiled, 16, "tma", 32)
    span, started = {}, threading.Event()

    def solve():
        torch.cuda.set_device(0)
        with torch.cuda.stream(torch.cuda.Stream()):
            started.set()
            span["begin"] = time.perf_counter()
            picuda.evolve_(dest, compiled, rho, (0.0, 2.5), steps=16000)
            span["end"] = time.perf_counter()

    t = threading.Thread(target=solve)
    t.start()
    started.wait()
    time.sleep(0.1)
    with torch.cuda.stream(torch.cuda.Stream()):
        t0 = time.perf_counter()
        picuda.apply_element_major_(Y, compiled, X)
        torch.cuda.current_stream().synchronize()
        took = time.perf_counter() - t0
        began_inside = "end" not in span
    t.join()
    torch.cuda.synchronize()
    total = span["end"] - span["begin"]
    assert began_inside and total > 0.3
    assert took < 0.15 * total, (took, total)
    assert torch.equal(Y, ref)
