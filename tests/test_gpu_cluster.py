"""Krylov cycles of the smallest job sets, which run as one thread-block cluster of up to 16 blocks,
against the graph of step kernels: the same bits, at one block, at the cluster's largest size and
just past it, with one job and with several."""
import numpy as np
import pytest

import picuda
from tests import models as M

pytestmark = pytest.mark.gpu

EXC = np.array([[0, 0], [0, 1]])


# FP64 blocks: 2, 3, 8, 13, 16 and 19 for the single jobs (a chunk of 32 entries each, and one)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("sizes", [(1,), (4,), (9,), (11,), (12,), (13,), (1, 2), (3, 6, 7)])
def test_cluster_cycle_equals_step_kernels(lib_built, sizes, precision):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    targets, general = [M.scan_model(N, 0.9, 0.3, 0.1) for N in sizes], M.general(5, 2)
    alg = picuda.ExpvAlgorithm(precision=precision, krylovdim=12)
    rho = [picuda.iid_pure_state(x.basis, np.array([0.28, 0.96j])) for x in targets + [general]]
    kw = dict(algorithm=alg, saveat=0.05, observables={"exc": EXC}, return_info=True)
    n = len(targets)
    ra, fa, ia = picuda.solve_dynamics_batch(targets, rho[:n], (0.0, 0.1), **kw)
    rb, fb, ib = picuda.solve_dynamics_batch(targets + [general], rho, (0.0, 0.1), **kw)
    for k in range(n):
        assert np.array_equal(fa[k], fb[k])
        assert np.array_equal(ra[k].values["exc"], rb[k].values["exc"])
        assert ia[k]["operator_applications"] == ib[k]["operator_applications"]
