"""The persistent Arnoldi recurrence with more basis vectors than one round of threads sums at four lanes a
value (64 complex ones): complex and real ground-state solves of up to 95 columns against the dense spectrum's
lowest values and the kernels launched one by one (eigenvalues of a basis orthogonal to a few eps: 1e-11)."""
import numpy as np
import pytest

import qudrip_gb300 as q
from qudrip_gb300 import chains

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("imag", [True, False])
@pytest.mark.parametrize("L,n,kdim", [(9, 4, 95), (11, 5, 70), (8, 4, 66), (13, 6, 80), (6, 3, 19)])
def test_many_vectors_equal_the_separate_kernels(ctx, monkeypatch, L, n, kdim, imag):
    spec, ham = chains.xxz_chain(L, 1.0, 0.7, True, np.linspace(-0.6, 0.8, L))
    sec = q.Sector(spec.index, [q.getNset(spec.index) == n])
    H = sec.lower(ham)
    rng = np.random.default_rng(L)
    x = rng.normal(size=sec.dim) + (1j * rng.normal(size=sec.dim) if imag else 0.0)
    psi = q.getState(sec, 1)
    got = {}
    for form in ("one", "split"):
        monkeypatch.setenv("QD_KRYLOV_STEP", form)
        psi.set(0, x)
        s = q.Arnoldi.getSolver(sec, kdim)
        s.getGroundState(H, psi, 0, -1)
        got[form] = (s.eigenvalues().copy(), psi.get(0))
    assert len(got["one"][0]) == len(got["split"][0])
    assert np.abs(got["one"][0] - got["split"][0]).max() < 1e-11
    assert abs(abs(np.vdot(got["one"][1], got["split"][1])) - 1.0) < 1e-10
