"""Trace balance of the FP64 level sweep with a free entry: z_f = (beta - sum t z) / t_f over the values
that were stored, so t^H z is beta up to the roundings of that one sum.

A thread adds up to ceil(entries / 128) products, a block sum of at most 16 additions follows, then a
subtraction, a division and the product t_f z_f here: (ceil(entries / 128) + 20) roundings of sum t |z|.
What beta itself is off by is measured in numpy, as its change under relative perturbations of one
rounding of the tables and the right-hand side, and counted 16 times."""
import math

import numpy as np
import pytest

import picuda
from tests import models as M
from tests.level_sweep_eval import sweep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("N", [30, 61, 100, 128])
def test_trace_of_the_sweep_is_beta(lib_built, N, seed):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    model = M.btc_c3(N, 1.0)
    P = picuda.level_preconditioner(picuda.compile(model), coords="reference", operator_scale=0.9)
    T = picuda.level_preconditioner_tables(model, coords="reference", operator_scale=0.9)
    assert T["mode"] == 0
    c0 = T["chain0_ent"]
    idx = T["elem"][c0:T["lev_ent"][T["chain_lev"][T["chain0"] + 1]]]
    r = M.random_state_vector(len(model.basis), seed)
    z = torch.empty(len(r), dtype=torch.complex128, device="cuda")
    P.apply(z, torch.from_numpy(r).cuda())
    tz = T["t0"] * z.cpu().numpy()[idx]
    trace = complex(math.fsum(tz.real), math.fsum(tz.imag))

    def beta(tables, rhs):  # with t the unit vector of the free entry the sweep leaves beta there
        t = np.zeros(len(idx))
        t[T["free_ent"] - c0] = 1.0
        return sweep({**tables, "t0": t}, rhs, 0.9)[T["elem"][T["free_ent"]]]

    rng = np.random.default_rng(seed)
    u = 2.0**-53

    def off(x):
        return np.asarray(x) * (1.0 + u * rng.uniform(-1.0, 1.0, np.shape(x)))

    ref = beta(T, r)
    moved = abs(beta({**T, **{k: off(T[k]) for k in ("W", "A", "C", "G")}}, off(r)) - ref)
    tol = (math.ceil(len(idx) / 128) + 20) * u * np.abs(tz).sum() + 16 * moved
    assert abs(trace - ref) <= tol
