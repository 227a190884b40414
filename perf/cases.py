"""What this engine's users have it do, as cases that a timer can run.

Each kind is one program's use of the public API:

  ground     a Lanczos ground state of a spin chain (getLanczosSolver): the README's XY chain, XXZ
             chains with and without fields, per-bond couplings, a ring with a flux (complex values),
             on the stored matrix or matrix-free
  hermitian  Hermitian::LanczosSolver on a Hubbard chain, the start of the dissipative programs
  arnoldi    the convergence loop of the Arnoldi ground-state solver on a 2D Heisenberg cluster
  quench     Krylov real-time steps of a Hubbard chain with observables accumulated at every step
             (McManager), Hermitian or with the no-jump damping of a dissipative chain
  evolve     Krylov real-time steps of a spin chain, full orthogonalisation (Arnoldi::getSolver)
  short      many real-time steps by the short-recurrence exponential (lanczos_evolve)
  batch      a disorder sweep: many ground states in one call (batch_lanczos)
  traj       quantum-jump trajectories of the dissipative Hubbard chain (traj_run)
  lower      a new operator on a chain: sector, `ham >> chain`, a product and an energy

Krylov dimensions of the solvers that do not reorthogonalise stay at 3 per site (5 for the
Hubbard chain): the lowest level is converged there and spurious copies have not come up yet.
"""
import math

import numpy as np
import torch

import qudrip_gb300 as q
from qudrip_gb300 import _capi as A
from qudrip_gb300 import chains


def listed():
    return [
        # the example program of a Hubbard quench: the smallest calls, where latency counts
        {"name": "quench-hubbard-L4", "kind": "quench", "L": 4, "nup": 2, "ndo": 2, "gamma": 0.0, "steps": 5,
         "m": 20, "dt": 0.05},
        # the no-jump evolution of the dissipative Hubbard chain: complex, not Hermitian
        {"name": "quench-damped-L8", "kind": "quench", "L": 8, "nup": 4, "ndo": 4, "gamma": 0.1, "steps": 10,
         "m": 30, "dt": 0.01},
        # an evolution request of the serving mix at its largest size, by the reference's algorithm
        {"name": "evolve-fields-L22", "kind": "evolve", "L": 22, "model": "fields", "m": 16, "dt": 0.05, "steps": 2},
        # the same kind of request as the mixed form serves it
        {"name": "short-xxz-L20", "kind": "short", "L": 20, "model": "xxz", "m": 32, "dt": 0.25, "steps": 20},
        # the README's program
        {"name": "ground-xy-L16", "kind": "ground", "L": 16, "model": "xy", "product": "csr"},
        # the headline workload
        {"name": "ground-xxz-L24", "kind": "ground", "L": 24, "model": "xxz", "product": "csr"},
        # couplings that differ bond by bond, without a stored matrix
        {"name": "ground-bonds-mfree-L20", "kind": "ground", "L": 20, "model": "bonds", "product": "mfree"},
        # the initial state of the dissipative program
        {"name": "hermitian-hubbard-L8", "kind": "hermitian", "L": 8, "nup": 4, "ndo": 4},
        # the 2D program's convergence loop
        {"name": "arnoldi-heisenberg-4x4", "kind": "arnoldi", "nx": 4, "ny": 4, "m": 60, "add": 10},
        # a disorder sweep
        {"name": "batch-fields-96", "kind": "batch", "n": 96, "Lmin": 14, "Lmax": 18, "steps": 80},
        # a part of the jump-trajectory ensemble
        {"name": "traj-hubbard-L8", "kind": "traj", "L": 8, "nup": 4, "ndo": 4, "ntraj": 2048, "steps": 100,
         "m": 30, "dt": 0.01, "gamma": 0.1},
        # a new point of a parameter scan
        {"name": "lower-xxz-L20", "kind": "lower", "L": 20, "model": "fields"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["quench", "evolve", "short", "ground", "ground", "hermitian", "arnoldi", "batch", "traj",
                       "lower"])
    if kind == "quench":
        L = rng.randint(3, 9)
        return {"kind": kind, "L": L, "nup": rng.randint(max(1, L // 2 - 1), L // 2 + 1),
                "ndo": rng.randint(max(1, L // 2 - 1), L // 2), "gamma": rng.choice([0.0, 0.1, 0.3]),
                "steps": rng.randint(2, 12), "m": rng.randint(12, 30), "dt": round(rng.uniform(0.01, 0.06), 3)}
    if kind == "evolve":
        return {"kind": kind, "L": rng.randint(10, 22), "model": rng.choice(["xy", "xxz", "fields", "bonds", "flux"]),
                "m": rng.randint(12, 24), "dt": round(rng.uniform(0.02, 0.06), 3), "steps": rng.randint(1, 4)}
    if kind == "short":
        return {"kind": kind, "L": rng.randint(10, 20), "model": rng.choice(["xy", "xxz", "fields", "bonds", "flux"]),
                "m": rng.randint(24, 32), "dt": round(rng.uniform(0.05, 0.25), 3), "steps": rng.randint(4, 30)}
    if kind == "ground":
        return {"kind": kind, "L": rng.randint(10, 22), "model": rng.choice(["xy", "xxz", "fields", "bonds", "flux"]),
                "product": rng.choice(["csr", "csr", "mfree"])}
    if kind == "hermitian":
        L = rng.randint(6, 9)
        return {"kind": kind, "L": L, "nup": rng.randint(L // 2 - 1, L // 2 + 1), "ndo": rng.randint(L // 2 - 1, L // 2)}
    if kind == "arnoldi":
        nx, ny = rng.choice([(3, 4), (2, 6), (2, 7), (3, 6), (4, 4), (2, 9), (4, 5)])
        return {"kind": kind, "nx": nx, "ny": ny, "m": rng.randint(30, 80), "add": rng.randint(5, 20)}
    if kind == "batch":
        lo = 2 * rng.randint(5, 8)
        c = {"kind": kind, "n": _log_int(rng, 8, 160), "Lmin": lo, "Lmax": min(18, lo + 2 * rng.randint(0, 2)),
             "steps": rng.randint(50, 90)}
        most = max(work(x)["bytes"] for x in listed())
        while work(c)["bytes"] > most:
            c["n"] -= 1
        return c
    if kind == "traj":
        L = rng.randint(4, 8)
        return {"kind": kind, "L": L, "nup": L // 2, "ndo": L // 2, "ntraj": _log_int(rng, 32, 2048),
                "steps": _log_int(rng, 10, 100), "m": rng.randint(12, 30), "dt": round(rng.uniform(0.005, 0.05), 3),
                "gamma": round(rng.uniform(0.05, 0.5), 2)}
    return {"kind": "lower", "L": rng.randint(8, 22), "model": rng.choice(["xy", "xxz", "fields", "bonds", "flux"])}


# ---------------------------------------------------------------- the physics, shared by the engine's call and exact()
def _spin_parameters(case, seed):
    """Per bond (i, j, hop amplitude of S+_i S-_j, J_z) and per site h; drawn from the seed."""
    L, model = case["L"], case["model"]
    rng = np.random.Generator(np.random.PCG64(seed))
    jz = float(rng.uniform(0.2, 1.8))
    if model == "xy":
        return [(i, i + 1, 1.0, None) for i in range(L - 1)], None
    if L == 24:
        jz = 1.0
    bonds = [(i, (i + 1) % L, 0.5, jz) for i in range(L)]
    h = None
    if model == "fields":
        h = rng.uniform(-1.0, 1.0, L)
    elif model == "bonds":
        bonds = [(i, j, float(rng.uniform(0.3, 0.7)), float(rng.uniform(0.5, 1.5))) for i, j, _, _ in bonds]
    elif model == "flux":
        phi = float(rng.uniform(0.3, 1.2))
        bonds = [(i, j, 0.5 * complex(math.cos(phi / L), math.sin(phi / L)), z) for i, j, _, z in bonds]
    return bonds, h


def _spin_operator(L, bonds, h):
    pre = q.getQbits(L)
    gc, ga, gz = q.getBoseGate(pre), q.getBoseGate(pre), q.getBoseGate(pre)
    gc << 0.5 * (q.pauli_x + q.II * q.pauli_y)
    ga << 0.5 * (q.pauli_x - q.II * q.pauli_y)
    gz << 0.5 * q.pauli_z
    ham = q.getEmptyOperator()
    for i, j, t, z in bonds:
        ham = ham + t * (gc(i) * ga(j)) + complex(t).conjugate() * (gc(j) * ga(i))
        if z is not None:
            ham = ham + z * (gz(i) * gz(j))
    if h is not None:
        for i in range(L):
            ham = ham + float(h[i]) * gz(i)
    return pre, [q.getNset(pre) == L // 2], ham


def _spin(case, seed):
    return _spin_operator(case["L"], *_spin_parameters(case, seed))


def _cluster_bonds(nx, ny):
    lat = q.Lattice([(i, j) for i in range(nx) for j in range(ny)], [(nx, 0), (0, ny)])
    return [(i, int(lat(lat(i) + np.array(a))), 0.5, 1.0) for i in range(lat.N()) for a in ((1, 0), (0, 1))]


def _hubbard(case):
    spec, ham = chains.hubbard_chain(case["L"], case["nup"], case["ndo"], 4.0, -1.0)
    if case.get("gamma"):
        gate = q.getHopFermiGate(spec.index)
        for s in range(2 * case["L"]):
            ham = ham + (-0.5j * case["gamma"]) * gate(s, s)
    return spec, ham


def _start(dim, seed, imag):
    rng = np.random.Generator(np.random.PCG64(seed + 1000))
    v = rng.uniform(-1.0, 1.0, dim).astype(np.complex128)
    if imag:
        v += 1j * rng.uniform(-1.0, 1.0, dim)
    return v / np.linalg.norm(v)


class _Column:
    def __init__(self, psi, t):
        self.psi = psi
        self.__cuda_array_interface__ = {"shape": (psi.dim,), "typestr": "<c16", "data": (psi.device_ptr(t), False),
                                         "version": 3, "strides": None}


def _view(psi, t):
    """Column t of a state, in place; the view keeps the state, whose memory it is, alive."""
    v = torch.as_tensor(_Column(psi, t), device="cuda")
    v.psi = psi
    return v


# ---------------------------------------------------------------- prepare and run
def _batch_sizes(case):
    span = range(case["Lmin"], case["Lmax"] + 1, 2)
    return [span[i % len(span)] for i in range(case["n"])]


def _batch_instance(case, seed, i, L):
    rng = np.random.Generator(np.random.PCG64([seed, i]))
    return [(a, (a + 1) % L, 0.5, 1.0) for a in range(L)], rng.uniform(-2.0, 2.0, L), rng


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        hams, v0s = [], []
        for i, L in enumerate(_batch_sizes(case)):
            bonds, h, rng = _batch_instance(case, seed, i, L)
            pre, cons, ham = _spin_operator(L, bonds, h)
            hams.append(q.Constrain(pre, *cons).lower(ham))
            v0s.append(rng.uniform(-1.0, 1.0, hams[-1].dim))
        return {"case": case, "hams": hams, "v0s": v0s}
    if kind == "traj":
        spec, ham = _hubbard(dict(case, gamma=0.0))
        sec = q.Constrain(spec.index, *spec.constraints)
        psi = q.getState(sec, 1)
        psi.set(0, _start(sec.dim, seed, False))
        q.Hermitian.LanczosSolver(sec, min(5 * case["L"], sec.dim // 2)).getGroundState(sec.lower(ham), psi, 0)
        psi0 = psi.get(0)
        heff = sec.lower(_hubbard(case)[1])
        return {"case": case, "heff": heff, "psi0": psi0 / np.linalg.norm(psi0), "seed": seed}
    if kind in ("quench", "hermitian"):
        spec, ham = _hubbard(case)
        sec = q.Constrain(spec.index, *spec.constraints)
    elif kind == "arnoldi":
        pre, cons, ham = _spin_operator(case["nx"] * case["ny"], _cluster_bonds(case["nx"], case["ny"]), None)
        sec = q.Constrain(pre, *cons)
    else:
        pre, cons, ham = _spin(case, seed)
        sec = q.Constrain(pre, *cons)
    nt = {"quench": case.get("steps", 0) + 1, "evolve": case.get("steps", 0) + 1}.get(kind, 2)
    psi = q.getState(sec, nt)
    s = {"case": case, "sec": sec, "psi": psi, "view": [_view(psi, t) for t in range(nt)]}
    evolves = kind in ("quench", "evolve", "short", "lower")
    # a solve overwrites column 0: its start waits in the last column
    psi.set(0 if evolves else nt - 1, _start(sec.dim, seed, evolves))
    if kind == "lower":
        s["cons"], s["pre"], s["ham"] = cons, pre, ham
        return s
    s["H"] = sec.lower(ham)
    if kind == "quench":
        L = case["L"]
        gate = q.getHopFermiGate(spec.index)
        s["docc"] = [sec.lower(chains.docc_operator(L, i, spec.index)) for i in range(L)]
        s["current"] = [sec.lower(1j * gate(i + 1, i) - 1j * gate(i, i + 1)) for i in range(L - 1)]
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "batch":
        out = q.batch_lanczos(s["hams"], s["v0s"], case["steps"])
        # the Krylov eigenvalue and the norm are computed in 32 bits, the refined energy in 64
        return {"krylov": out[:, 0].astype(np.float32), "energy": out[:, 1].copy(),
                "norm": out[:, 2].astype(np.float32), "act": out[:, 3].astype(np.int64)}
    if kind == "traj":
        L = case["L"]
        mean, err, _ = q.traj_run(s["heff"], s["psi0"], case["ntraj"], case["steps"], case["dt"], case["gamma"],
                                  s["seed"], case["m"], range(2 * L), [(i, i + L) for i in range(L)])
        # the states and the records are 32 bits wide
        return {"mean": mean.astype(np.float32), "err": err.astype(np.float32)}
    sec, psi = s["sec"], s["psi"]
    if kind == "lower":
        sec = q.Constrain(s["pre"], *s["cons"])
        H = sec.lower(s["ham"])
        q.apply(H, psi, 0, psi, 1)
        return {"dim": sec.range(), "nnz": H.nnz, "real": H.is_real, "hermitian": H.is_hermitian,
                "energy": np.array(psi.eval(0, H)), "product": s["view"][1]}
    H = s["H"]
    if kind == "ground":
        A.call("qd_state_copy", psi.handle, 1, psi.handle, 0)
        spmv = A.QD_SPMV_MATRIX_FREE if case["product"] == "mfree" else A.QD_SPMV_CSR
        solver = q.Arnoldi.getLanczosSolver(sec, 3 * case["L"], spmv=spmv)
        solver.getGroundState(H, psi(0), 0)
        return {"energy": solver.eigenvalues()[0], "evals": solver.eigenvalues(), "psi": s["view"][0]}
    if kind == "hermitian":
        A.call("qd_state_copy", psi.handle, 1, psi.handle, 0)
        solver = q.Hermitian.LanczosSolver(sec, 5 * case["L"])
        solver.getGroundState(H, psi, 0)
        return {"energy": solver.eigenvalues()[0], "evals": solver.eigenvalues(), "psi": s["view"][0]}
    if kind == "arnoldi":
        A.call("qd_state_copy", psi.handle, 1, psi.handle, 0)
        solver = q.Arnoldi.getSolver(sec, case["m"])
        solver.convergeEV(1, 0.0)
        while solver.act_dim() < case["m"]:
            solver.getGroundState(H, psi(0), 0, case["add"])
            if solver.error() < 1e-10:
                break
        return {"energy": solver.eigenvalues()[0], "evals": solver.eigenvalues(), "psi": s["view"][0]}
    if kind == "short":
        q.lanczos_evolve(H, psi, 0, 1, case["dt"], case["m"], case["steps"])
        return s["view"][1]
    solver = q.Arnoldi.getSolver(sec, case["m"])
    if kind == "evolve":
        for t in range(case["steps"]):
            solver.evolve(H, psi(t), t, case["dt"])
        return s["view"][1:]
    mc = q.McManager(psi.nt(), psi)
    for name in ("docc", "current"):
        mc.addObs(name, len(s[name]))
        for i, op in enumerate(s[name]):
            mc.updateMatrix(name, i, op)
    for t in range(psi.nt()):
        if t > 0:
            solver.evolve(H, psi(t - 1), t - 1, case["dt"])
        mc.incrAllObs(t)
    mc.normAll()
    return {"psi": s["view"][1:], "docc": mc.data["docc"], "current": mc.data["current"]}


# ---------------------------------------------------------------- work
def _spin_counts(L, nup, nb, diagonal):
    dim = math.comb(L, nup)
    return dim, 2 * nb * math.comb(L - 2, nup - 1) + (dim if diagonal else 0)


def _hubbard_counts(case):
    L, a, b = case["L"], case["nup"], case["ndo"]
    da, db = math.comb(L, a), math.comb(L, b)
    hops = lambda n: 2 * (L - 1) * (math.comb(L - 2, n - 1) if 0 < n < L else 0)  # noqa: E731
    return da * db, hops(a) * db + hops(b) * da + da * db


def _counts(case):
    if case["kind"] in ("quench", "hermitian", "traj"):
        return _hubbard_counts(case)
    if case["kind"] == "arnoldi":
        n = case["nx"] * case["ny"]
        return _spin_counts(n, n // 2, 2 * n, True)
    L, xy = case["L"], case["model"] == "xy"
    return _spin_counts(L, L // 2, L - 1 if xy else L, not xy)


def work(case):
    """Per product the matrix (4-byte columns and its values) and the vector in and out; per stored basis
    vector one read for each use that the algorithm makes of it; flops as multiplies and adds."""
    kind = case["kind"]
    if kind == "batch":
        by = fl = 0
        for L in _batch_sizes(case):
            dim, nnz = _spin_counts(L, L // 2, L, True)
            k = case["steps"]
            by += k * (4 * nnz + 16 * dim) + 8 * dim * k * (k + 1) // 2 + 8 * dim
            fl += k * (2 * nnz + 12 * dim) + 4 * dim * k * (k + 1) // 2
        return {"bytes": by, "flops": fl}
    dim, nnz = _counts(case)
    cplx = kind in ("quench", "evolve", "short") or case.get("model") == "flux"
    vb, vf = (16, 4) if cplx else (8, 1)
    mvb, mvf = (16, 4) if case.get("model") == "flux" or case.get("gamma") else (8, 2 if cplx else 1)
    product = (4 + mvb) * nnz + 2 * vb * dim
    pflops = 2 * mvf * nnz
    if kind == "traj":
        steps = case["ntraj"] * case["steps"]
        return {"bytes": 12 * nnz + 8 * dim + 4 * case["L"] * steps, "flops": steps * 6 * (4 * nnz + 16 * dim)}
    if kind == "lower":
        return {"bytes": 8 * dim + (4 + mvb) * nnz + 2 * 16 * dim, "flops": 4 * mvf * nnz}
    if kind == "ground" or kind == "hermitian":
        k = 3 * case["L"] if kind == "ground" else 5 * case["L"]
        if case.get("product") == "mfree":
            product = (8 + 8 + 2 * vb) * dim
        return {"bytes": k * (product + vb * dim) + k * vb * dim + 32 * dim,
                "flops": k * (pflops + 14 * vf * dim)}
    if kind == "short":
        k = case["m"] - 1
        return {"bytes": case["steps"] * (k * (product + vb * dim) + k * vb * dim + 32 * dim),
                "flops": case["steps"] * k * (pflops + 14 * vf * dim)}
    k = case["m"] if kind == "arnoldi" else case["m"] - 1
    # every previous vector is read for its projection and once more to be taken out
    one = {"bytes": k * product + vb * dim * k * (k + 1) + k * vb * dim,
           "flops": k * pflops + 4 * vf * dim * k * (k + 1) // 2}
    n = 1 if kind == "arnoldi" else case["steps"]
    obs = (case["steps"] + 1) * 2 * case["L"] * 16 * dim if kind == "quench" else 0
    return {"bytes": n * one["bytes"] + obs, "flops": n * one["flops"] + obs // 4}


# ---------------------------------------------------------------- exact
class _Plain:
    """y = H x in plain torch, 64 bits, term by term on the sector's states."""

    def __init__(self, states, dev):
        self.states, self.dev, self.terms = states, dev, []
        self.diag = torch.zeros(len(states), dtype=torch.complex128, device=dev)

    def rank(self, st):
        return torch.searchsorted(self.states, st)

    def hop(self, a, b, t, sign=False):
        """t c+_a c_b (sign: fermions, with the string between the two sites); the conjugate is its own term."""
        s = self.states
        rows = torch.nonzero((((s >> a) & 1) == 1) & (((s >> b) & 1) == 0)).flatten()  # the row has a, not b
        col = s[rows] ^ ((1 << a) | (1 << b))
        v = torch.ones(len(rows), dtype=torch.float64, device=self.dev)
        if sign:
            for k in range(min(a, b) + 1, max(a, b)):
                v = v * (1 - 2 * ((s[rows] >> k) & 1))
        self.terms.append((rows, self.rank(col), v * t if isinstance(t, complex) else v * float(t)))

    def __call__(self, x):
        y = self.diag.to(x.dtype) * x if x.is_complex() else self.diag.real * x
        for rows, cols, v in self.terms:
            y.index_add_(0, rows, v.to(x.dtype) * x[cols])
        return y


def _bit(s, k):
    return ((s >> k) & 1).to(torch.float64)


def _plain_spin(L, bonds, h, dev):
    s = torch.arange(1 << L, device=dev)
    n = torch.zeros_like(s)
    for k in range(L):
        n += (s >> k) & 1
    P = _Plain(s[n == L // 2].contiguous(), dev)
    for i, j, t, z in bonds:
        P.hop(i, j, t)
        P.hop(j, i, t.conjugate() if isinstance(t, complex) else t)
        if z is not None:
            P.diag += z * _spin_z(P.states, i) * _spin_z(P.states, j)
    if h is not None:
        for i in range(L):
            P.diag += float(h[i]) * _spin_z(P.states, i)
    return P


def _spin_z(s, i):
    # gz << pauli_z / 2 on bit i: the matrix's row 0 is the empty bit
    return 0.5 - _bit(s, i)


def _plain_hubbard(case, dev):
    L = case["L"]

    def half(n):
        return [s for s in range(1 << L) if bin(s).count("1") == n]

    s = torch.tensor([u | (d << L) for d in half(case["ndo"]) for u in half(case["nup"])], device=dev)
    P = _Plain(torch.sort(s).values, dev)
    for o in (0, L):
        for i in range(L - 1):
            P.hop(i + 1 + o, i + o, -1.0, True)
            P.hop(i + o, i + 1 + o, -1.0, True)
    for i in range(L):
        P.diag += 4.0 * _bit(P.states, i) * _bit(P.states, i + L)
    if case.get("gamma"):
        P.diag += -0.5j * case["gamma"] * sum(_bit(P.states, k) for k in range(2 * L))
    return P


def _krylov_lowest(P, v0, k):
    """Eigenvalues of P on the Krylov space of dimension k, fully orthogonalised."""
    n = len(v0)
    V = torch.zeros((k, n), dtype=v0.dtype, device=v0.device)
    V[0] = v0 / torch.linalg.vector_norm(v0)
    a, b = [], []
    for i in range(k):
        w = P(V[i])
        a.append(torch.vdot(V[i], w).real)
        for _ in range(2):
            w = w - V[: i + 1].T @ (V[: i + 1].conj() @ w)
        b.append(torch.linalg.vector_norm(w))
        if float(b[-1]) < 1e-10 or i + 1 == k:
            break
        V[i + 1] = w / b[-1]
    T = torch.diag(torch.stack(a))
    if len(a) > 1:
        off = torch.stack(b[: len(a) - 1])
        T = T + torch.diag(off, 1) + torch.diag(off, -1)
    return torch.linalg.eigvalsh(T.cpu()).numpy()


def _propagate(P, x, dt):
    """exp(-i P dt) x by Taylor steps of small norm."""
    bound = float(P.diag.abs().max()) + sum(float(v.abs().max()) for _, _, v in P.terms)
    n = max(1, math.ceil(bound * dt / 0.5))
    for _ in range(n):
        t, y = x, x
        for k in range(1, 24):
            t = P(t) * (-1j * dt / n / k)
            y = y + t
        x = y
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "traj":
        return None  # decided by the engine's own random stream
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "batch":
        ev = []
        for i, L in enumerate(_batch_sizes(case)):
            bonds, h, rng = _batch_instance(case, seed, i, L)
            P = _plain_spin(L, bonds, h, dev)
            v0 = torch.from_numpy(rng.uniform(-1.0, 1.0, len(P.states))).to(dev)
            ev.append(_krylov_lowest(P, v0, case["steps"])[0])
        return {"krylov": np.array(ev), "energy": np.array(ev), "norm": None, "act": None}
    if kind in ("quench", "hermitian"):
        P = _plain_hubbard(case, dev)
    elif kind == "arnoldi":
        P = _plain_spin(case["nx"] * case["ny"], _cluster_bonds(case["nx"], case["ny"]), None, dev)
    else:
        P = _plain_spin(case["L"], *_spin_parameters(case, seed), dev)
    dim = len(P.states)
    evolves = kind in ("quench", "evolve", "short", "lower")
    x = torch.from_numpy(_start(dim, seed, evolves)).to(dev)
    if kind == "lower":
        y = P(x)
        return {"dim": None, "nnz": None, "real": None, "hermitian": None,
                "energy": np.array(complex(torch.vdot(x, y))), "product": y}
    if kind in ("ground", "hermitian"):
        v0 = x if case.get("model") == "flux" else x.real.contiguous()
        # K products span K vectors; the solver's sign of the state is its own
        ev = _krylov_lowest(P, v0, 3 * case["L"] if kind == "ground" else 5 * case["L"] + 1)
        return {"energy": np.array(ev[0]), "evals": ev, "psi": None}
    if kind == "arnoldi":
        ev = _krylov_lowest(P, x.real.contiguous(), case["m"])
        return {"energy": np.array(ev[0]), "evals": None, "psi": None}  # the loop ends on its own error
    if kind == "short":
        for _ in range(case["steps"]):
            x = _propagate(P, x, case["dt"])
        return x
    states = [x]
    for _ in range(case["steps"]):
        y = _propagate(P, states[-1] / torch.linalg.vector_norm(states[-1]), case["dt"])
        states.append(y)
    if kind == "evolve":
        return states[1:]
    L = case["L"]
    docc = np.zeros((case["steps"] + 1, L), dtype=np.complex128)
    cur = np.zeros((case["steps"] + 1, L - 1), dtype=np.complex128)
    for i in range(L):
        d = _bit(P.states, i) * _bit(P.states, i + L)
        for t, y in enumerate(states):
            docc[t, i] = float((d * (y.abs() ** 2)).sum())
    for i in range(L - 1):
        C = _Plain(P.states, dev)
        C.hop(i + 1, i, 1j, True)
        C.hop(i, i + 1, -1j, True)
        for t, y in enumerate(states):
            cur[t, i] = complex(torch.vdot(y, C(y)))
    return {"psi": states[1:], "docc": docc, "current": cur}
