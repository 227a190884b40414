"""The Gram-Schmidt passes over a basis in memory (sectors too large for the persistent recurrence, and
every sector when the kernels are launched one by one) against the oracle and the short recurrence: ragged
tiles, one to three chunks of vectors, Hermitian and not, early breakdown, and the copies left out (served
requests).  A state is orthogonalised to a few eps per vector: m * 10 eps < 1e-13; the tests allow 1e-12."""
import numpy as np
import pytest

import oracle as O
import qudrip_gb300 as q
from qudrip_gb300 import chains

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.fixture(autouse=True)
def one_by_one(monkeypatch):
    monkeypatch.setenv("QD_KRYLOV_STEP", "split")


def start(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=n) + 1j * rng.normal(size=n)
    return x / np.linalg.norm(x)


def chain(L, n, damped=False):
    spec, ham = chains.xxz_chain(L, 1.0, 0.7, True, np.linspace(-0.6, 0.8, L))
    pre = spec.index
    if damped:
        gz = q.getBoseGate(pre)
        gz << 0.5 * q.pauli_z
        for i in range(L):
            ham = ham + (-0.02j * (i + 1)) * gz(i)
    return q.SectorSpec(pre, [q.getNset(pre) == n]), ham


@pytest.mark.parametrize("damped", [False, True])
@pytest.mark.parametrize("L,n,m", [(6, 3, 2), (8, 4, 33), (9, 4, 20), (10, 5, 33), (12, 6, 9), (13, 6, 33)])
def test_evolution_equals_the_oracle(ctx, L, n, m, damped):
    spec, ham = chain(L, n, damped)
    sec = q.Sector(spec.index, spec.constraints)
    H = sec.lower(ham)
    x = start(sec.dim, L)
    psi = q.getState(sec, 1)
    psi.set(0, 3.0 * x)  # the start vector is normalised
    solver = q.Arnoldi.getSolver(sec, m)
    for _ in range(2):
        solver.evolve_inplace(H, psi, 0, 0.07)
        ref, _ = O.Ham(O.Sector(spec), ham).arnoldi_evolve(x, 0.07, m)
        got = psi.get(0)
        assert np.linalg.norm(got - ref) < TOL
        x = got


def test_large_sector_equals_the_short_recurrence(ctx):
    spec, ham = chain(20, 10)  # 184,756 rows: 128-row tiles, the last one ragged
    sec = q.Sector(spec.index, spec.constraints)
    H = sec.lower(ham)
    x = start(sec.dim, 3)
    psi = q.getState(sec, 2)
    psi.set(0, x)
    psi.set(1, x)
    q.Arnoldi.getSolver(sec, 30).evolve_inplace(H, psi, 0, 0.05)
    q.lanczos_evolve(H, psi, 1, 1, 0.05, 30)
    assert np.linalg.norm(psi.get(0) - psi.get(1)) < TOL


def test_ground_state_grown_over_three_chunks(ctx):
    spec, ham = chain(11, 5)
    sec = q.Sector(spec.index, spec.constraints)
    H = sec.lower(ham)
    psi = q.getState(sec, 1)
    psi.set(0, start(sec.dim, 1))
    solver = q.Arnoldi.getSolver(sec, 75)
    for _ in range(3):  # 25, 50 and 75 columns
        solver.getGroundState(H, psi(0), 0, 25)
    w, v = np.linalg.eigh(H.scipy().toarray())
    assert abs(solver.eigenvalues()[0] - w[0]) < 1e-11
    assert abs(abs(np.vdot(v[:, 0], psi.get(0))) - 1.0) < 1e-10
