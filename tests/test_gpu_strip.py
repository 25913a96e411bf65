"""Strip apply (merged coefficient planes) against the host-lowered stencil tables.

Per output entry at most 11 products are summed, each of rounded factors, so the result lies
within 32 rounding units of the sum of the products' magnitudes."""
import numpy as np
import pytest

import picuda
from oracle import pi_oracle as O
from tests import models as M
from tests.stencil_eval import evaluate

pytestmark = pytest.mark.gpu

S = picuda.spin_matrices(2)
# every kernel variant: 0, 1, 3, 5, 6, 8 gain positions with and without a drive
FAMILIES = {
    "collective": dict(hamiltonian=0.7 * S["jx"], collective_emission=0.3),
    "btc": dict(hamiltonian=0.7 * S["jx"], collective_emission=0.3, dephasing=0.2),
    "ensemble": dict(hamiltonian=0.3 * S["jz"] + 1.2 * S["jx"], emission=0.2, dephasing=0.1, collective_emission=0.05),
    "pumped": dict(hamiltonian=0.3 * S["jz"] + 1.2 * S["jx"], emission=0.2, pumping=0.1),
    "all": dict(hamiltonian=0.3 * S["jz"] + 1.2 * S["jx"], emission=0.2, pumping=0.1, dephasing=0.1),
    "undriven": dict(hamiltonian=0.4 * S["jz"], emission=0.2, dephasing=0.1),
    "undriven_all": dict(emission=0.2, pumping=0.3, dephasing=0.1, collective_dephasing=0.05),
    "unitary": dict(hamiltonian=0.3 * S["jz"] + 1.2 * S["jx"]),
}


@pytest.fixture(scope="module")
def torch_cuda(lib_built):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _bound(basis, table, coef, x):
    return evaluate(basis, table, np.abs(coef).astype(np.complex128), np.abs(x)).real


# n^2 = 64 and 256 end on a full warp (N = 7, 15); odd sizes leave a partial one
@pytest.mark.parametrize("N", [1, 2, 7, 15, 34])
@pytest.mark.parametrize("family", sorted(FAMILIES))
def test_strip_apply_matches_tables(torch_cuda, family, N):
    torch = torch_cuda
    for sectors in (None, [(N, 0)], [(N - k, k) for k in range(0, N // 2 + 1, 2)]):
        model = picuda.qubit_ensemble_model(picuda.PIBasis(N, 2, sectors=sectors), **FAMILIES[family])
        compiled = picuda.compile(model)
        assert compiled.info["batched_kernel"] == 2
        n = len(model.basis)
        for adjoint, apply in ((False, picuda.apply_), (True, picuda.apply_adjoint_)):
            table, coef = picuda.stencil_tables(model, adjoint=adjoint)
            for ncols in (1, 3, 17, 65):
                X = np.stack([M.random_state_vector(n, 7 * c + N) for c in range(ncols)])
                xd = torch.from_numpy(X if ncols > 1 else X[0]).cuda()
                y = apply(torch.full_like(xd, float("nan")), compiled, xd).cpu().numpy().reshape(ncols, n)
                for c in {0, ncols // 2, ncols - 1}:
                    ref = evaluate(model.basis, table, coef, X[c])
                    tol = 32 * np.finfo(float).eps * _bound(model.basis, table, coef, X[c])
                    assert (np.abs(y[c] - ref) <= tol).all(), (sectors, adjoint, ncols, c)


@pytest.mark.parametrize("N", [1, 2, 7, 15, 34])
@pytest.mark.parametrize("family", sorted(FAMILIES))
def test_strip_apply_f32_matches_tables(torch_cuda, family, N):
    torch = torch_cuda
    model = picuda.qubit_ensemble_model(N, **FAMILIES[family])
    compiled = picuda.compile(model)
    n = len(model.basis)
    root = np.repeat(model.basis.multiplicity_scales(), np.array(model.basis.dims) ** 2)  # z = root x
    table, coef = picuda.stencil_tables(model)
    for ncols in (1, 3, 17, 65):
        X = np.stack([M.random_state_vector(n, 5 * c + N) for c in range(ncols)]).astype(np.complex64)
        xd = torch.from_numpy(X if ncols > 1 else X[0]).cuda()
        for coords, scale in (("reference", np.ones(n)), ("population", root)):
            y = picuda.apply_(torch.full_like(xd, float("nan")), compiled, xd, precision="fp32", coords=coords)
            y = y.cpu().numpy().reshape(ncols, n)
            for c in {0, ncols // 2, ncols - 1}:
                x = X[c].astype(np.complex128) / scale
                ref = scale * evaluate(model.basis, table, coef, x)
                tol = 32 * np.finfo(np.float32).eps * scale * _bound(model.basis, table, coef, x)
                assert (np.abs(y[c] - ref) <= tol).all(), (coords, ncols, c)


@pytest.mark.parametrize("family", ["undriven", "all", "btc"])
def test_strip_engine_and_rk4_match_oracle(torch_cuda, family):
    model = picuda.qubit_ensemble_model(11, **FAMILIES[family])
    compiled = picuda.compile(model)
    oplan = O.Plan(M.to_oracle(model))
    psi = np.array([0.6, 0.8j])
    rho = picuda.iid_pure_state(model.basis, psi)
    L = lambda v: O.apply(oplan, v)  # noqa: E731
    ref, _ = O.krylov_expv(L, rho.data.copy(), 0.3)
    got = picuda.krylov_expv(compiled, rho, 0.3)
    assert np.abs(got - ref).max() <= 1e-9 * np.abs(ref).max()
    x, h = rho.data.copy(), 0.3 / 50
    for _ in range(50):
        k1 = L(x)
        k2 = L(x + (h / 2) * k1)
        k3 = L(x + (h / 2) * k2)
        k4 = L(x + h * k3)
        x = x + (h / 6) * (k1 + 2 * k2 + 2 * k3 + k4)
    got = picuda.time_evolve(compiled, rho, (0.0, 0.3), steps=50).data
    assert np.abs(got - x).max() <= 1e-12 * np.abs(x).max()


def test_first_apply_inside_a_graph_capture(torch_cuda):
    """A plan's planes are built on its first FP64 apply, also when that one is being captured."""
    torch = torch_cuda
    model = M.ensemble_c2(21)
    compiled = picuda.compile(model)
    x = torch.from_numpy(M.random_state_vector(len(model.basis), 3)).cuda()
    y, ref = torch.zeros_like(x), torch.zeros_like(x)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        picuda.apply_(y, compiled, x)
    g.replay()
    picuda.apply_(ref, compiled, x)
    torch.cuda.synchronize()
    assert torch.equal(y, ref) and bool((ref != 0).any())
