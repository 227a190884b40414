"""Open Arnoldi ground-state solves (getGroundState called again to grow the Krylov space): what ends
them and what a grown call reports."""
import numpy as np
import pytest

import qudrip_gb300 as q
from qudrip_gb300 import _capi as A
from qudrip_gb300 import chains

pytestmark = pytest.mark.gpu

KDIM, ADD = 30, 10


def hubbard():
    spec, ham = chains.hubbard_chain(4, 2, 2, 4.0, -1.0, periodic=True)  # 36 rows
    sec = q.Sector(spec.index, spec.constraints)
    return sec, ham


def xxz(L=10):
    spec, ham = chains.xxz_chain(L, 1.0, 0.7, True, np.linspace(-1, 1, L))  # 252 rows: several blocks
    return q.Sector(spec.index, spec.constraints), ham


def start(sec):
    psi = q.getState(sec, 1)
    psi.set(0, q.start_vector(sec.dim, 4).astype(complex))
    return psi


@pytest.mark.parametrize("system", [hubbard, xxz])
@pytest.mark.parametrize("factor", [2.0, 1j])
@pytest.mark.parametrize("form", ["one", "split"])
def test_scaling_the_operator_ends_its_open_solve(ctx, monkeypatch, system, factor, form):
    if form == "split":
        monkeypatch.setenv("QD_KRYLOV_STEP", "split")
    sec, ham = system()
    H = sec.lower(ham)
    psi = start(sec)
    solver = q.Arnoldi.getSolver(sec, KDIM)
    solver.getGroundState(H, psi, 0, ADD)
    H.scale(factor)
    with pytest.raises(A.QDError) as e:
        solver.getGroundState(H, psi, 0, ADD)
    assert e.value.code == A.QD_ERR_INVALID
    # a new solve on the scaled operator is one on an operator scaled before it was ever solved
    psi = start(sec)
    a = q.Arnoldi.getSolver(sec, KDIM)
    a.getGroundState(H, psi, 0, ADD)
    fresh = sec.lower(ham)
    fresh.scale(factor)
    psi2 = start(sec)
    b = q.Arnoldi.getSolver(sec, KDIM)
    b.getGroundState(fresh, psi2, 0, ADD)
    assert np.array_equal(a.eigenvalues(), b.eigenvalues())
    assert np.array_equal(psi.get(0), psi2.get(0))


@pytest.mark.parametrize("system", [hubbard, xxz])
@pytest.mark.parametrize("form", ["one", "split"])
def test_a_grown_solve_reports_the_change_of_its_lowest_eigenvalue(ctx, monkeypatch, system, form):
    if form == "split":
        monkeypatch.setenv("QD_KRYLOV_STEP", "split")
    sec, ham = system()
    H = sec.lower(ham)
    psi = start(sec)
    solver = q.Arnoldi.getSolver(sec, KDIM)
    last = 0.0
    for _ in range(3):
        r = solver.getGroundState(H, psi, 0, ADD)
        assert r.err == abs(r.ritz_value - last)  # |lambda_0| first, then |lambda_0 - previous lambda_0|
        last = r.ritz_value
