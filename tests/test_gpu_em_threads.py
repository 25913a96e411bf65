"""Element-major applies of several threads on one compiled model, each thread on a stream and on
more source batches of its own than the plan keeps tensor maps for: every launch uses the maps of
its own batch, also when another thread displaces them in between."""
import threading

import pytest

import picuda
from tests import models as M

pytestmark = pytest.mark.gpu


def test_first_apply_of_a_new_thread(lib_built):
    """A thread whose first CUDA call is an apply of a new batch, pinned to the TMA kernel."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    compiled = picuda.compile(M.ensemble_c2(25))
    x = torch.randn((len(compiled.basis), 16), dtype=torch.complex64, device="cuda")
    y, ref = torch.zeros_like(x), torch.zeros_like(x)
    picuda.select_element_major_kernel(compiled, 16, "tma", 32)
    torch.cuda.synchronize()
    errors = []

    def worker():
        try:
            picuda.apply_element_major_(y, compiled, x)
        except Exception as err:
            errors.append(repr(err))

    t = threading.Thread(target=worker)
    t.start()
    t.join()
    picuda.apply_element_major_(ref, compiled, x)
    torch.cuda.synchronize()
    assert not errors, errors
    assert torch.equal(y, ref)


@pytest.mark.parametrize("ncols", [16, 64])  # narrow and full blocks
def test_threads_with_many_batches(lib_built, ncols):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    compiled = picuda.compile(M.ensemble_c2(25))
    n = len(compiled.basis)
    g = torch.Generator(device="cuda").manual_seed(7)
    threads, batches, rounds = 6, 5, 40
    xs = [[torch.randn((n, ncols), dtype=torch.complex64, device="cuda", generator=g) for _ in range(batches)]
          for _ in range(threads)]
    picuda.select_element_major_kernel(compiled, ncols, "tma", 32)
    refs = [[picuda.apply_element_major_(torch.empty_like(x), compiled, x) for x in row] for row in xs]
    ys = [[torch.full_like(x, float("nan")) for x in row] for row in xs]
    torch.cuda.synchronize()
    start, errors = threading.Barrier(threads), []

    def worker(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait()
                for _ in range(rounds):
                    for x, y in zip(xs[k], ys[k]):
                        picuda.apply_element_major_(y, compiled, x)
        except Exception as err:  # pragma: no cover - reported below
            errors.append(repr(err))

    pool = [threading.Thread(target=worker, args=(k,)) for k in range(threads)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for k in range(threads):
        for y, ref in zip(ys[k], refs[k]):
            assert torch.equal(y, ref)
