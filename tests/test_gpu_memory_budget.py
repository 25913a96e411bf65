"""memory_budget of compile: coefficient planes that do not fit are not laid out, and every call that
would use them gives the same result from the general kernels.

Per output entry at most 11 products are summed, so two orders of summation differ by at most 64
rounding units of the sum of the products' magnitudes (32 for each side, as against the tables)."""
import numpy as np
import pytest

import picuda
from tests import models as M
from tests.stencil_eval import evaluate

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda(lib_built):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def table_bytes(model):
    """Device memory of the tables that a plan cannot do without."""
    held = picuda.compile(model).info["device_bytes"]
    try:
        return picuda.compile(model, memory_budget=held - 1).info["device_bytes"]
    except picuda.PiArgumentError:  # nothing optional so far
        return held


def test_planes_within_the_budget_only(torch_cuda):
    torch = torch_cuda
    model = M.ensemble_c2(40)
    n = len(model.basis)
    free = picuda.compile(model)
    own = table_bytes(model)
    table, coef = picuda.stencil_tables(model)
    X = np.stack([M.random_state_vector(n, c) for c in range(5)])
    bound = np.stack([evaluate(model.basis, table, np.abs(coef).astype(complex), np.abs(x)).real for x in X])
    x = torch.from_numpy(X).cuda()
    y = picuda.apply_(torch.empty_like(x), free, x).cpu().numpy()
    used = free.info["device_bytes"]
    assert used >= own + 7 * 8 * n  # two planes and five gain positions
    # room for the tables, for the strip items as well, for all but a byte of the planes
    for budget in (own, own + 3 * n, used - 1):
        tight = picuda.compile(model, memory_budget=budget)
        for form in (x, x[0]):
            got = picuda.apply_(torch.full_like(form, float("nan")), tight, form).cpu().numpy().reshape(-1, n)
            m = len(got)
            assert (np.abs(got - y[:m]) <= 64 * 2.0**-52 * bound[:m]).all()
        host = np.empty_like(X)
        picuda.apply_(host, tight, X)
        assert (np.abs(host - y) <= 64 * 2.0**-52 * bound).all()
        assert tight.info["device_bytes"] <= budget
    exact = picuda.compile(model, memory_budget=used)
    assert torch.equal(picuda.apply_(torch.empty_like(x), exact, x).cpu(), torch.from_numpy(y))
    assert exact.info["device_bytes"] == used
    # FP32 planes take half the room
    half = picuda.compile(model, memory_budget=used - 1)
    x32 = x.to(torch.complex64)
    ref32 = picuda.apply_(torch.empty_like(x32), free, x32, precision="fp32")
    assert torch.equal(picuda.apply_(torch.empty_like(x32), half, x32, precision="fp32"), ref32)
    assert own < half.info["device_bytes"] < used
    with pytest.raises(picuda.PiArgumentError):
        picuda.compile(model, memory_budget=own - 1)


def test_adjoint_and_solvers_under_a_tight_budget(torch_cuda):
    torch = torch_cuda
    model = M.ensemble_c2(24)
    n = len(model.basis)
    free = picuda.compile(model)
    own = table_bytes(model)
    tight = picuda.compile(model, memory_budget=own)
    x = torch.from_numpy(M.random_state_vector(n, 9)).cuda()
    a = picuda.apply_adjoint_(torch.empty_like(x), free, x)
    b = picuda.apply_adjoint_(torch.empty_like(x), tight, x)
    table, coef = picuda.stencil_tables(model, adjoint=True)
    bound = evaluate(model.basis, table, np.abs(coef).astype(complex), x.abs().cpu().numpy().astype(complex)).real
    assert (np.abs((a - b).cpu().numpy()) <= 64 * 2.0**-52 * bound).all()
    assert tight.adjoint().info["device_bytes"] <= own
    rho = picuda.computational_product_state(model.basis, 2)
    # solvers of the same tolerance: the RK4 steps round differently, the Krylov steps stop at 1e-10
    for solve, tol in ((lambda c: picuda.time_evolve(c, rho, (0.0, 0.2), steps=40).data, 1e-12),
                       (lambda c: picuda.krylov_expv(c, rho, 0.2), 1e-9)):
        p, q = solve(free), solve(tight)
        assert np.abs(p - q).max() <= tol * np.abs(p).max()
    assert tight.info["device_bytes"] <= own


@pytest.mark.parametrize("N", [8, 97, 160])
def test_first_fp64_apply_allocates_nothing(torch_cuda, N):
    """compile reserves the planes of a first FP64 apply; those of FP32 take half of it."""
    torch = torch_cuda
    model = M.ensemble_c2(N)
    n = len(model.basis)
    for dtype, precision in ((torch.complex128, "fp64"), (torch.complex64, "fp32")):
        compiled = picuda.compile(model)
        held = compiled.info["device_bytes"]
        assert held >= table_bytes(model) + 7 * 8 * n
        x = torch.zeros(n, dtype=dtype, device="cuda")
        picuda.apply_(torch.empty_like(x), compiled, x, precision=precision)
        assert compiled.info["device_bytes"] == held
        x = torch.zeros(n, dtype=torch.complex128, device="cuda")
        picuda.apply_adjoint_(torch.empty_like(x), compiled, x)
        assert compiled.info["device_bytes"] == held  # the adjoint has its own
    assert compiled.adjoint().info["device_bytes"] >= table_bytes(model) + 7 * 8 * n


def test_unused_reserves_are_given_back(torch_cuda):
    """What an allocation that fails does first: the room of plans that have not used it is freed, those
    plans allocate later, and a plan that has used its room keeps it."""
    torch = torch_cuda
    reclaim = picuda.load_library()._ZN6picuda16reclaim_reservesEv
    model = M.ensemble_c2(30)
    used, unused = picuda.compile(model), picuda.compile(model)
    x = torch.from_numpy(M.random_state_vector(len(model.basis), 1)).cuda()
    ref = picuda.apply_(torch.empty_like(x), used, x)
    held = used.info["device_bytes"]
    assert unused.info["device_bytes"] == held
    assert reclaim() & 0xFF
    assert used.info["device_bytes"] == held and unused.info["device_bytes"] == table_bytes(model)
    for compiled in (used, unused):
        assert torch.equal(picuda.apply_(torch.empty_like(x), compiled, x), ref)
    gone = picuda.compile(model)
    gone.close()
    reclaim()  # a closed plan is no longer listed


def test_mixed_solves_round_alike_under_any_budget(torch_cuda):
    """FP32 steps by strips whatever the budget, so that every engine schedule gives the same bits."""
    model = M.ensemble_c2(30)
    rho = picuda.computational_product_state(model.basis, 2)
    alg = picuda.ExpvAlgorithm(krylovdim=20, precision="mixed")
    out = {}
    try:
        for budget in (None, table_bytes(model)):
            for schedule in ("auto", "per_tile", 1):
                picuda.set_engine_schedule(schedule)
                compiled = picuda.compile(model, memory_budget=budget)
                _, finals = picuda.solve_dynamics_batch([compiled], [rho], (0.0, 0.2), saveat=0.1, algorithm=alg)
                out[budget, schedule] = np.asarray(finals[0])
    finally:
        picuda.set_engine_schedule("auto")
    ref = out[None, "auto"]
    for key, got in out.items():
        assert np.array_equal(got, ref), key
