"""A Krylov cycle as one cooperative launch (small sets of canonical plans) against the graph of
step kernels that larger or general sets run: the same bits, for every chunk size of the FP64
reductions, with early stops and with short cycles."""
import numpy as np
import pytest

import picuda
from tests import models as M

pytestmark = pytest.mark.gpu

EXC = np.array([[0, 0], [0, 1]])


@pytest.fixture(scope="module")
def torch_cuda(lib_built):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


# dims 10, 165, 969, 12,341, 32,016 and 79,079: 128 to 1024 elements per FP64 chunk
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("N,m", [(3, 30), (8, 4), (8, 30), (16, 50), (40, 17), (55, 30), (76, 8)])
def test_cycle_equals_step_kernels(torch_cuda, N, m, precision):
    target, general = M.scan_model(N, 0.9, 0.3, 0.1), M.general(5, 2)  # a general plan keeps the graph
    alg = picuda.ExpvAlgorithm(precision=precision, krylovdim=m)
    rho = [picuda.iid_pure_state(x.basis, np.array([0.28, 0.96j])) for x in (target, general)]
    t = 0.02 if m < 8 else 0.1
    kw = dict(algorithm=alg, saveat=t, observables={"exc": EXC}, return_info=True)
    ra, fa, ia = picuda.solve_dynamics_batch([target], rho[:1], (0.0, 2 * t), **kw)
    rb, fb, ib = picuda.solve_dynamics_batch([target, general], rho, (0.0, 2 * t), **kw)
    assert np.array_equal(fa[0], fb[0])
    assert np.array_equal(ra[0].values["exc"], rb[0].values["exc"])
    assert ia[0]["operator_applications"] == ib[0]["operator_applications"]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_gmres_cycle_equals_step_kernels(torch_cuda, precision):
    models = [M.driven_c1(7), M.driven_c1(12), M.driven_c1(16)]
    alg = picuda.GMRESAlgorithm(krylovdim=50, maxiter=3000, precision=precision)
    kw = dict(algorithm=alg, return_info=True, raise_on_failure=False)
    a, ia = picuda.stationary_state_batch(models, **kw)
    b, ib = picuda.stationary_state_batch(models + [M.general(4, 1)], **kw)
    for x, y, p, q in zip(a, b, ia, ib):
        assert p["converged"] and p["iterations"] == q["iterations"]
        assert np.array_equal(x.data, y.data)
