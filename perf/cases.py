"""Performance cases of the qubit-ensemble Liouvillian and its solvers on one GPU.

Every case is work that a user of `picuda` asks for through its public entry points: the
Liouvillian action on one vector or a batch (`apply_`, `apply_adjoint_`,
`apply_element_major_`), fixed-step RK4 (`evolve_`), Krylov dynamics with streamed observables
(`solve_dynamics`), a batched parameter scan (`solve_dynamics_batch`) and steady states
(`stationary_state`).  `exact` evaluates the same quantities in 64 bits from the closed-form
matrix elements of collective spins and of local jumps on Schur blocks (B. A. Chase and
J. M. Geremia, Phys. Rev. A 78, 052101 (2008)), with plain torch and no code of the package.
"""
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = Path(__file__).resolve().parents[1] / "permutationalinvariantdynamics.jl_gb300"
if str(_PKG) not in sys.path:
    sys.path.insert(0, str(_PKG))


# --------------------------------------------------------------------------------------
# The cases
# --------------------------------------------------------------------------------------

def listed():
    return [
        # One action on the smallest ensemble of the configurations (dim 165): a user's own
        # integrator around apply!, where the launch is all there is.
        dict(name="apply_f64_N8", kind="apply", N=8, cols=1, model="driven", precision="fp64"),
        # The headline workload: 128 resident vectors in the reference's matrix layout.
        dict(name="apply_f64_N120_x128", kind="apply", N=120, cols=128, model="ensemble", precision="fp64"),
        # One adjoint action at the largest steady-state size (dim 1.37 million): left
        # eigenvectors, duality checks, sensitivities.
        dict(name="adjoint_f64_N200", kind="adjoint", N=200, cols=1, model="ensemble", precision="fp64"),
        # A ragged batch of an odd size with pumping, FP32 in the reference's layout.
        dict(name="apply_f32_N97_x37", kind="apply", N=97, cols=37, model="driven", precision="fp32"),
        # The FP32 action on a batch stored element by element.
        dict(name="apply_em_f32_N120_x128", kind="apply_em", N=120, cols=128, model="ensemble", precision="fp32"),
        # The default dynamics algorithm on the large time evolution: one saved interval.
        dict(name="rk4_f64_N120", kind="rk4", N=120, model="ensemble", precision="fp64", steps=64),
        # The smallest time evolution: t in [0, 4] saved every 0.1 with one observable.
        dict(name="expv_f64_N8", kind="expv", N=8, model="driven", precision="fp64", intervals=40, dt=0.1),
        # The large time evolution, four saved intervals with two streamed observables, plain
        # and mixed precision.
        dict(name="expv_f64_N120", kind="expv", N=120, model="ensemble", precision="fp64", intervals=4, dt=0.05),
        dict(name="expv_mixed_N120", kind="expv", N=120, model="ensemble", precision="mixed", intervals=4, dt=0.05),
        # A parameter scan over instances of uneven size (N drawn from 20..160).
        dict(name="scan_mixed_x24", kind="scan", count=24, Nmin=20, Nmax=160, precision="mixed", intervals=2, dt=0.05),
        # A steady state by the reference's own restarted GMRES.
        dict(name="steady_f64_N16", kind="steady", N=16, model="driven", precision="fp64", krylovdim=50),
        # The largest steady state (boundary time crystal with dephasing), preconditioned,
        # mixed precision.
        dict(name="steady_mixed_N200", kind="steady", N=200, model="btc", precision="mixed", krylovdim=50),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["apply", "apply", "adjoint", "apply_em", "rk4", "expv", "expv", "scan", "steady"])
    model = rng.choice(["ensemble", "ensemble", "driven", "tilted"])
    if kind in ("apply", "adjoint"):
        N = _log_int(rng, 4, 200)
        most = max(1, min(160, 38_000_000 // _dim(N)))
        return dict(kind=kind, N=N, cols=_log_int(rng, 1, most), model=model, precision=rng.choice(["fp64", "fp32"]))
    if kind == "apply_em":
        N = _log_int(rng, 8, 160)
        most = max(1, min(128, 38_000_000 // _dim(N) // 2))
        return dict(kind=kind, N=N, cols=2 * _log_int(rng, 1, most), model=rng.choice(["ensemble", "driven"]),
                    precision="fp32")
    if kind == "rk4":
        return dict(kind=kind, N=_log_int(rng, 6, 130), model=model, precision=rng.choice(["fp64", "mixed"]),
                    steps=rng.choice([50, 64, 100]))
    if kind == "expv":
        return dict(kind=kind, N=_log_int(rng, 6, 120), model=model, precision=rng.choice(["fp64", "mixed"]),
                    intervals=rng.randint(1, 4), dt=rng.choice([0.05, 0.1]))
    if kind == "scan":
        lo = rng.randint(12, 60)
        return dict(kind=kind, count=rng.randint(3, 24), Nmin=lo, Nmax=rng.randint(lo + 10, 120),
                    precision=rng.choice(["fp64", "mixed"]), intervals=rng.randint(1, 2), dt=0.05)
    if rng.random() < 0.5:
        return dict(kind="steady", N=rng.randint(5, 15), model="driven", precision="fp64", krylovdim=rng.randint(45, 60))
    return dict(kind="steady", N=rng.randint(40, 199), model="btc", precision=rng.choice(["fp64", "mixed"]),
                krylovdim=rng.randint(40, 60))


def _dim(N):
    return sum((N - 2 * k + 1) ** 2 for k in range(N // 2 + 1))


# Rates of one model, drawn around the repository's configurations.
def _rates(case, rng, N):
    u = rng.uniform
    r = dict(hz=0.0, hx=0.0, hy=0.0, emission=0.0, dephasing=0.0, pumping=0.0, collective=0.0)
    if case["kind"] == "scan":  # the parameter scan's ranges
        r.update(hx=u(0.2, 2.0), emission=u(0.05, 0.5), dephasing=u(0.0, 0.2), collective=1.0 / N)
    elif case["model"] == "btc":  # drive below, at and above the collective rate 1 / N
        kappa = 1.0 / N
        r.update(hx=rng.choice([0.5, 1.0, 2.0]) * kappa * u(0.98, 1.02), dephasing=0.01 * u(0.9, 1.1), collective=kappa)
    elif case["kind"] == "steady":
        r.update(hx=u(0.95, 1.05), emission=u(0.48, 0.55))
    elif case["model"] == "driven" and case["kind"] == "expv":
        r.update(hx=u(0.9, 1.1), emission=u(0.45, 0.55))
    elif case["model"] == "driven":
        r.update(hx=u(0.5, 0.9), hz=u(0.1, 0.3), emission=u(0.1, 0.2), pumping=u(0.01, 0.05))
    else:
        r.update(hz=u(0.25, 0.35), hx=u(1.0, 1.3), emission=u(0.15, 0.25), dephasing=u(0.05, 0.15),
                 collective=u(0.04, 0.06) / N)
        if case["model"] == "tilted":  # a drive with a phase
            r.update(hy=u(0.2, 0.4))
    return r


def _model(rates, N):
    import picuda
    s = picuda.spin_matrices(2)
    h = rates["hz"] * s["jz"] + rates["hx"] * s["jx"] + rates["hy"] * s["jy"]
    return picuda.qubit_ensemble_model(N, hamiltonian=h, emission=rates["emission"], dephasing=rates["dephasing"],
                                       pumping=rates["pumping"], collective_emission=rates["collective"])


def _instances(case, seed):
    """(N, rates) of every model of a case."""
    rng = random.Random(1000003 * seed + 17)
    if case["kind"] == "scan":
        sizes = random.Random(7).choices(range(case["Nmin"], case["Nmax"] + 1), k=case["count"])
        return [(N, _rates(case, rng, N)) for N in sizes]
    return [(case["N"], _rates(case, rng, case["N"]))]


def _coords(case):
    return "population" if case["kind"] == "apply_em" else "reference"


def _batch(case, seed):
    """Complex normal vectors, the Krylov and probe vectors of the solvers."""
    dim, cols = _dim(case["N"]), case["cols"]
    dt = torch.complex128 if case["precision"] == "fp64" else torch.complex64
    g = torch.Generator(device="cuda").manual_seed(seed + 11)
    shape = (dim, cols) if case["kind"] == "apply_em" else ((dim,) if cols == 1 else (cols, dim))
    return torch.randn(shape, dtype=dt, device="cuda", generator=g)


def _psi(seed):
    """One qubit's pure state: mostly excited, with some coherence."""
    rng = random.Random(31 * seed + 5)
    th, ph = rng.uniform(0.0, 0.5), rng.uniform(0.0, 2 * math.pi)
    return np.array([math.sin(th) * complex(math.cos(ph), math.sin(ph)), math.cos(th)], dtype=np.complex128)


# --------------------------------------------------------------------------------------
# prepare and run
# --------------------------------------------------------------------------------------

def prepare(case, seed):
    import picuda
    kind = case["kind"]
    inst = _instances(case, seed)
    compiled = [picuda.compile(_model(r, N)) for N, r in inst]
    c = compiled[0]
    st = dict(case=case, compiled=compiled)
    if kind in ("apply", "adjoint", "apply_em"):
        st["x"] = _batch(case, seed)
        st["y"] = torch.empty_like(st["x"])
        if kind == "adjoint":
            c.adjoint()
    elif kind == "rk4":
        rho = picuda.iid_pure_state(c.basis, _psi(seed))
        st["src"] = torch.from_numpy(rho.data).cuda()
        st["dest"] = torch.empty_like(st["src"])
    elif kind == "expv":
        st["rho"] = picuda.iid_pure_state(c.basis, _psi(seed))
        s = picuda.spin_matrices(2)
        st["obs"] = {"Jz": picuda.collective_operator(c.basis, s["jz"]),
                     "JpJm": picuda.collective_operator(c.basis, s["jp"] @ s["jm"])}
    elif kind == "scan":
        s = picuda.spin_matrices(2)
        st["rho"] = [picuda.computational_product_state(m.basis, 2) for m in compiled]
        st["obs"] = [{"Jz": picuda.collective_operator(m.basis, s["jz"])} for m in compiled]
    elif case["model"] == "btc":  # preconditioned, in population coordinates
        P = picuda.level_preconditioner(c, coords="population")
        st["alg"] = picuda.GMRESAlgorithm(krylovdim=case["krylovdim"], maxiter=2000, precision=case["precision"],
                                          preconditioner=P)
    else:
        st["alg"] = picuda.GMRESAlgorithm(krylovdim=case["krylovdim"], maxiter=5000, precision=case["precision"])
    return st


def run(st):
    import picuda
    case, c = st["case"], st["compiled"][0]
    kind = case["kind"]
    if kind == "apply":
        return picuda.apply_(st["y"], c, st["x"], precision=case["precision"])
    if kind == "adjoint":
        return picuda.apply_adjoint_(st["y"], c, st["x"], precision=case["precision"])
    if kind == "apply_em":
        return picuda.apply_element_major_(st["y"], c, st["x"], coords="population")
    if kind == "rk4":
        return picuda.evolve_(st["dest"], c, st["src"], (0.0, 0.05), steps=case["steps"], precision=case["precision"])
    if kind == "expv":
        alg = picuda.ExpvAlgorithm(krylovdim=30, precision=case["precision"])
        r = picuda.solve_dynamics(c, st["rho"], (0.0, case["intervals"] * case["dt"]), algorithm=alg,
                                  saveat=case["dt"], observables=st["obs"], save_states=False)
        return {k: r.values[k] for k in st["obs"]}
    if kind == "scan":
        alg = picuda.ExpvAlgorithm(krylovdim=30, precision=case["precision"])
        r, finals = picuda.solve_dynamics_batch(st["compiled"], st["rho"], (0.0, case["intervals"] * case["dt"]),
                                                algorithm=alg, saveat=case["dt"], observables=st["obs"])
        return {"values": [x.values["Jz"] for x in r], "finals": finals}
    # a residual of 1e-12 and below, so that the state is settled to ten digits and more
    atol, rtol = (2e-12, 2e-12) if case["model"] == "btc" else (1e-13, 2e-11)
    return picuda.stationary_state(c, algorithm=st["alg"], atol=atol, rtol=rtol).data


# --------------------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------------------

def _positions(case):
    """Stencil positions of an output entry: (complex or imaginary, real)."""
    if case["kind"] != "scan" and case["model"] == "btc":
        return 5, 4  # centre, drive; own (-1,-1), dephasing from the own and both neighbour sectors
    return 5, 8 if case["kind"] != "scan" and case["model"] == "driven" else 5


def _apply_flops(case):
    """Real operations per entry: the complex centre, four imaginary neighbours (two fused
    multiply-adds each) and the real gains."""
    _, real = _positions(case)
    return 2 * (4 + 4 * 2 + 2 * real)


def work(case):
    kind = case["kind"]
    b = 16 if case["precision"] == "fp64" else 8
    if kind in ("apply", "adjoint", "apply_em"):
        e = _dim(case["N"]) * case["cols"]
        return {"bytes": 2 * b * e, "flops": _apply_flops(case) * e}
    if kind == "rk4":  # the state in and out; four actions and the stage updates per step
        e = _dim(case["N"])
        return {"bytes": 2 * 16 * e, "flops": case["steps"] * 4 * (_apply_flops(case) + 8) * e}
    if kind in ("expv", "scan"):
        # one Krylov space of 30 per interval: an action, projections onto and updates by the
        # space built so far (8 + 8 operations per entry and vector), and the combination
        m = 30
        e = sum(_dim(N) for N, _ in _instances(case, 0))
        per = m * _apply_flops(case) + 16 * m * (m + 1) // 2 + 8 * m
        obs = 1 if kind == "scan" else 2
        return {"bytes": e * ((2 + obs) * 16 + case["intervals"] * b * 2 * m), "flops": case["intervals"] * per * e}
    # a steady state: some tens of preconditioned, or some hundreds of plain, GMRES steps
    e = _dim(case["N"])
    its = 60 if case["model"] == "btc" else 300
    return {"bytes": e * (16 + its * 2 * b), "flops": its * (_apply_flops(case) + 16 * 25) * e}


# --------------------------------------------------------------------------------------
# 64-bit values from the closed-form matrix elements
# --------------------------------------------------------------------------------------

class _Generator:
    """L as a list of gathers, y[e] = sum_k c_k[e] x[i_k[e]].  Sector k has J = N/2 - k and an
    n x n column-major block over m = J - row, m' = J - column.  population: entries are summed
    over the sector's f copies (z = sqrt(f) x); otherwise x = z / sqrt(f)."""

    def __init__(self, N, rates, population=False):
        dev = "cuda"
        ns = [N - 2 * k + 1 for k in range(N // 2 + 1)]
        offs = np.concatenate([[0], np.cumsum([n * n for n in ns])])
        self.dim = int(offs[-1])
        k = torch.repeat_interleave(torch.arange(len(ns)), torch.tensor([n * n for n in ns])).to(dev)
        off = torch.tensor(offs, device=dev)
        local = torch.arange(self.dim, device=dev) - off[k]
        n = N - 2 * k + 1
        a, b = local % n, local // n
        J = N / 2 - k.double()
        ma, mb = J - a, J - b
        self.terms = []

        def root(v):
            return v.clamp(min=0).sqrt()

        def add(dk, da, db, coef):
            # source sector k + dk at (a + da, b + db)
            ks = k + dk
            nsrc = N - 2 * ks + 1
            ia, ib = a + da, b + db
            ok = (ks >= 0) & (ks < len(ns)) & (ia >= 0) & (ib >= 0) & (ia < nsrc) & (ib < nsrc)
            i = torch.where(ok, off[ks.clamp(0, len(ns) - 1)] + ia + ib * nsrc, torch.zeros_like(ia))
            c = torch.as_tensor(coef, device=dev).to(torch.complex128).expand(self.dim)
            self.terms.append((i, torch.where(ok, c, torch.zeros_like(c)), ok))

        up = lambda m: root((J - m) * (J + m + 1))  # noqa: E731  <m+1|J+|m>
        dn = lambda m: root((J + m) * (J - m + 1))  # noqa: E731  <m-1|J-|m>
        r = rates
        em, ph, pu, co = r["emission"], r["dephasing"], r["pumping"], r["collective"]
        loss = sum(em * (N / 2 + m) + ph * N / 4 + pu * (N / 2 - m) + co * dn(m) ** 2 for m in (ma, mb))
        add(0, 0, 0, -1j * r["hz"] * (ma - mb) - 0.5 * loss)
        w = complex(r["hx"], -r["hy"]) / 2  # H = hz Jz + w J+ + conj(w) J-
        if w != 0:
            add(0, 1, 0, -1j * w * up(ma - 1))
            add(0, -1, 0, -1j * w.conjugate() * dn(ma + 1))
            add(0, 0, -1, 1j * w * up(mb))
            add(0, 0, 1, 1j * w.conjugate() * dn(mb))
        if co:
            add(0, -1, -1, co * dn(ma + 1) * dn(mb + 1))
        # local gains: sum_i s_q^i |J' m><J' m'| s_q^i+ lands in J' (A), J' - 1 (B) and J' + 1 (D)
        elements = {
            -1: (lambda j, m: root((j + m) * (j - m + 1)), lambda j, m: root((j + m) * (j + m - 1)),
                 lambda j, m: root((j - m + 1) * (j - m + 2))),
            0: (lambda j, m: m, lambda j, m: root((j + m) * (j - m)), lambda j, m: root((j + m + 1) * (j - m + 1))),
            1: (lambda j, m: root((j - m) * (j + m + 1)), lambda j, m: root((j - m) * (j - m - 1)),
                lambda j, m: root((j + m + 1) * (j + m + 2))),
        }
        kd, nd = k.double(), n.double()
        Js = J.clamp(min=0.25)
        for q, rate in ((-1, em), (0, ph), (1, pu)):
            if not rate:
                continue
            A, B, D = elements[q]
            sa, sb = ma - q, mb - q  # source magnetic numbers
            own = torch.where(J > 0, (1 + (kd / nd) * (2 * J + 1) / (J + 1)) / (2 * Js), torch.zeros_like(J))
            add(0, q, q, rate * own * A(J, sa) * A(J, sb))
            # from J' = J + 1 (sector k - 1): alpha' / (2 J' f') times sqrt(f' / f)
            c2 = (N - kd + 2) / (nd + 2) / (2 * (J + 1))
            fr = 1.0 if population else root(kd * (nd + 2) / (nd * (N - kd + 2)))
            add(-1, q + 1, q + 1, rate * c2 * fr * B(J + 1, sa) * B(J + 1, sb))
            # from J' = J - 1 (sector k + 1)
            c3 = (kd + 1) / (nd - 2).clamp(min=1) / (2 * Js)
            fr = 1.0 if population else root((nd - 2) * (N - kd + 1) / ((kd + 1) * nd))
            add(1, q - 1, q - 1, rate * c3 * fr * D(J - 1, sa) * D(J - 1, sb))

    def __call__(self, x):
        """L x along the last axis."""
        y = torch.zeros_like(x)
        for i, c, _ in self.terms:
            y += c * x[..., i]
        return y

    def adjoint(self, x):
        y = torch.zeros_like(x)
        for i, c, ok in self.terms:  # each term's map is one to one on its valid entries
            y[..., i[ok]] += c[ok].conj() * x[..., ok]
        return y


def _roots_of_f(N):
    """sqrt(f) per entry."""
    out = []
    for k in range(N // 2 + 1):
        f = math.comb(N, k) - (math.comb(N, k - 1) if k else 0)
        out += [math.sqrt(f)] * (N - 2 * k + 1) ** 2
    return torch.tensor(out, dtype=torch.float64, device="cuda")


def _iid(N, psi):
    v = np.array([math.sqrt(math.comb(N, a)) * psi[0] ** a * psi[1] ** (N - a) for a in range(N + 1)])
    x = torch.zeros(_dim(N), dtype=torch.complex128, device="cuda")
    x[: (N + 1) ** 2] = torch.from_numpy(np.outer(v, v.conj()).reshape(-1, order="F")).cuda()
    return x


def _observables(N):
    """{name: vector} with the value sum_e vector[e] z[e], z = sqrt(f) x."""
    jz = torch.zeros(_dim(N), dtype=torch.float64, device="cuda")
    one = torch.zeros_like(jz)
    o = 0
    for k in range(N // 2 + 1):
        n = N - 2 * k + 1
        d = o + torch.arange(n, device="cuda") * (n + 1)
        jz[d] = (N / 2 - k) - torch.arange(n, device="cuda", dtype=torch.float64)
        one[d] = 1.0
        o += n * n
    return {"Jz": jz, "JpJm": jz + N / 2 * one}


def _exponential(L, x, t, bound):
    """exp(t L) x by Taylor series on substeps of norm about two."""
    steps = max(1, int(math.ceil(t * bound / 2)))
    h = t / steps
    for _ in range(steps):
        term, y = x, x.clone()
        for p in range(1, 60):
            term = (h / p) * L(term)
            y += term
            if p % 5 == 0 and float(torch.linalg.vector_norm(term)) < 1e-18 * float(torch.linalg.vector_norm(y)):
                break
        x = y
    return x


def _bound(N, rates):
    J = N / 2
    return 2 * J * (abs(rates["hx"]) + abs(rates["hy"]) + abs(rates["hz"])) + N * (
        rates["emission"] + rates["pumping"] + rates["dephasing"]) * 2 + 2 * rates["collective"] * J * (J + 1)


def exact(case, seed):
    kind = case["kind"]
    inst = _instances(case, seed)
    N, rates = inst[0]
    if kind in ("apply", "adjoint", "apply_em"):
        L = _Generator(N, rates, population=_coords(case) == "population")
        x = _batch(case, seed)
        if kind == "apply_em":
            x = x.T
        cols = x.reshape(-1, x.shape[-1])
        out = torch.empty(cols.shape, dtype=torch.complex128, device="cuda")
        for i in range(0, cols.shape[0], 16):
            v = cols[i:i + 16].to(torch.complex128)
            out[i:i + 16] = L.adjoint(v) if kind == "adjoint" else L(v)
        out = out.reshape(x.shape)
        return out.T if kind == "apply_em" else out
    if kind == "rk4":
        if case["steps"] * _dim(N) > 64 * 500_000:
            return None
        L, x, h = _Generator(N, rates), _iid(N, _psi(seed)), 0.05 / case["steps"]
        for _ in range(case["steps"]):
            k1 = L(x)
            k2 = L(x + (h / 2) * k1)
            k3 = L(x + (h / 2) * k2)
            k4 = L(x + h * k3)
            x = x + (h / 6) * (k1 + 2 * k2 + 2 * k3 + k4)
        return x
    if kind == "expv":
        L, z = _Generator(N, rates, population=True), _iid(N, _psi(seed))
        obs = _observables(N)
        got = {k: [complex((v * z).sum())] for k, v in obs.items()}
        for _ in range(case["intervals"]):
            z = _exponential(L, z, case["dt"], _bound(N, rates))
            for k, v in obs.items():
                got[k].append(complex((v * z).sum()))
        return {k: np.array(v) for k, v in got.items()}
    if kind == "scan":
        values, finals = [], []
        for N, rates in inst:
            L, z = _Generator(N, rates, population=True), _iid(N, np.array([0.0, 1.0], dtype=np.complex128))
            jz = _observables(N)["Jz"]
            vals = [complex((jz * z).sum())]
            for _ in range(case["intervals"]):
                z = _exponential(L, z, case["dt"], _bound(N, rates))
                vals.append(complex((jz * z).sum()))
            values.append(np.array(vals))
            finals.append((z / _roots_of_f(N)).cpu().numpy())
        return {"values": values, "finals": finals}
    if _dim(N) > 1200:
        return None
    # L x = 0 with t^H x = 1, t the trace functional: (L + t t^H / |t|^2) x = t / |t|^2
    L = _Generator(N, rates)
    dense = L(torch.eye(L.dim, dtype=torch.complex128, device="cuda")).T
    obs = _observables(N)
    t = ((obs["JpJm"] - obs["Jz"]) * (2 / N) * _roots_of_f(N)).to(torch.complex128)
    v = t / torch.linalg.vector_norm(t) ** 2
    return torch.linalg.solve(dense + torch.outer(v, t.conj()), v).cpu().numpy()
