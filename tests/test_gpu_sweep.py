"""The level sweep at the sizes where its layout changes: one to three entries per lane of the
solving warp (levels of up to 32, 33, 64, 65 and 66 entries), chains shorter and longer than the
ring of level slots, with and without a free entry, against the numpy sweep of the exported tables.

A value passes through at most N + 1 levels, each adding a few roundings of the gains, the products
of multipliers and two scans: 16 (N + 8) roundings of the working precision, relative to the
largest entry.  Levels with a small pivot and the border's correction amplify the roundings of the
tables, the right-hand side and the arithmetic alike; how much is measured in numpy, as the change
under relative perturbations of one rounding in each of them, and counted 16 times."""
import numpy as np
import pytest

import picuda
from tests import models as M
from tests.level_sweep_eval import sweep

pytestmark = pytest.mark.gpu


def perturbed(T, r, eps, rng):
    """The sweep of tables and right-hand side with relative errors of up to eps in each entry."""
    def off(x):
        return np.asarray(x) * (1.0 + eps * rng.uniform(-1.0, 1.0, np.shape(x)))
    return sweep({**T, **{k: off(T[k]) for k in ("W", "A", "C", "G", "w0")}}, off(r), 0.9)


@pytest.mark.parametrize("coords,eps", [("population", 2.0**-24), ("reference", 2.0**-53)])
@pytest.mark.parametrize("regularization", [0.0, 0.3])
@pytest.mark.parametrize("N", [1, 6, 62, 65, 127, 128, 130])
def test_sweep_layout_edges(lib_built, N, regularization, coords, eps):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    model = M.btc_c3(N, 1.0)
    P = picuda.level_preconditioner(picuda.compile(model), coords=coords, operator_scale=0.9,
                                    regularization=regularization)
    T = picuda.level_preconditioner_tables(model, coords=coords, operator_scale=0.9, regularization=regularization)
    r = M.random_state_vector(len(model.basis), N)
    rd = torch.from_numpy(r).cuda()
    zd = torch.full_like(rd, float("nan"))
    P.apply(zd, rd)
    ref = sweep(T, r, 0.9)
    amplified = np.abs(perturbed(T, r, eps, np.random.default_rng(N)) - ref).max()
    assert np.abs(zd.cpu().numpy() - ref).max() <= 16 * ((N + 8) * eps * np.abs(ref).max() + amplified)
