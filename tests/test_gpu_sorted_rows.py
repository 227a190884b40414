"""The persistent Lanczos recurrence takes a block's rows in order of their length: sectors whose blocks hold
ragged numbers of rows, lengths up to and past the 63 told apart, and rows of the diagonal alone, against the
Arnoldi recurrence.  Both orthogonalise to a few eps a step: 1e-12."""
import numpy as np
import pytest

import qudrip_gb300 as q
from qudrip_gb300 import chains

pytestmark = pytest.mark.gpu


def pairs(L, n, reach, real):
    """Hops between all pairs of sites less than `reach` apart, site energies on the first half."""
    pre = q.getQbits(L)
    gc, ga, gz = q.getBoseGate(pre), q.getBoseGate(pre), q.getBoseGate(pre)
    gc << 0.5 * (q.pauli_x + q.II * q.pauli_y)
    ga << 0.5 * (q.pauli_x - q.II * q.pauli_y)
    gz << 0.5 * q.pauli_z
    ham = q.getEmptyOperator()
    for i in range(L):
        for j in range(i + 1, min(L, i + reach)):
            t = (0.3 + 0.05 * i + 0.02 * j) * (1.0 if real else 1.0 + 0.4j)
            ham = ham + t * (gc(i) * ga(j)) + np.conj(t) * (gc(j) * ga(i))
        if i < L // 2:
            ham = ham + (0.4 * i - 1.0) * gz(i)
    return q.SectorSpec(pre, [q.getNset(pre) == n]), ham


@pytest.mark.parametrize("L,n,reach,real", [
    (18, 9, 18, True),    # 48,620 rows of up to 82 entries
    (18, 8, 18, False),   # 43,758
    (20, 6, 2, False),    # 38,760 rows of 1 to 14
    (19, 9, 3, True),     # 92,378
    (40, 3, 40, True),    # 9,880 rows of 112: fewer rows a block than threads
])
def test_sorted_rows_equal_the_arnoldi_recurrence(ctx, L, n, reach, real):
    spec, ham = pairs(L, n, reach, real)
    sec = q.Sector(spec.index, spec.constraints)
    H = sec.lower(ham)
    rng = np.random.default_rng(L + n)
    x = rng.normal(size=sec.dim) + 1j * rng.normal(size=sec.dim)
    x /= np.linalg.norm(x)
    psi = q.getState(sec, 2)
    psi.set(0, x)
    psi.set(1, x)
    m, dt = 20, 0.02
    q.lanczos_evolve(H, psi, 0, 0, dt, m)
    q.Arnoldi.getSolver(sec, m).evolve_inplace(H, psi, 1, dt)
    assert np.linalg.norm(psi.get(0) - psi.get(1)) < 1e-12
