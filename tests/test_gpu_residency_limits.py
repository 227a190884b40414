"""The Arnoldi recurrence just below and above the rows that its persistent form keeps on the chip: which form
runs is told by its launches, and each is compared with something other than itself."""
import numpy as np
import pytest
import scipy.sparse.linalg as sla

import qudrip_gb300 as q
from qudrip_gb300 import chains

from test_gpu_persistent_krylov import TOL, damped_hubbard, fields

pytestmark = pytest.mark.gpu


def magnetised(L, n):
    spec, ham = chains.xxz_chain(L, 1.0, 0.7, True, np.linspace(-1, 1, L))
    return q.SectorSpec(spec.index, [q.getNset(spec.index) == n]), ham


# 38,760 rows: 323 a block of 120, with 34 vectors beside the exponential's matrix all but full
@pytest.mark.parametrize("make,resident", [(lambda: magnetised(20, 6), True), (lambda: fields(19), False),
                                           (lambda: damped_hubbard(10, 5, 5), False)])
def test_evolution_at_the_limit(ctx, make, resident):
    spec, ham = make()
    sec = q.Sector(spec.index, spec.constraints)
    H = sec.lower(ham)
    rng = np.random.default_rng(1)
    x = rng.normal(size=sec.dim) + 1j * rng.normal(size=sec.dim)
    x /= np.linalg.norm(x)
    st = q.getState(sec, 3)
    st.set(0, x)
    s = q.Arnoldi.getSolver(sec, 33)
    s.evolve(H, st(0), 0, 0.02)
    n0 = ctx.launches()
    s.evolve(H, st(0), 0, 0.02)
    assert (ctx.launches() - n0 <= 2) == resident
    assert s.act_dim() == 32
    # 32 columns at ||h H|| < 1: the truncation is far below rounding
    exact = sla.expm_multiply(-0.02j * H.scipy().tocsc(), x)
    if not H.is_hermitian:  # (the input is normalised, the output is not)
        assert np.linalg.norm(st.get(1)) < 1.0
    assert np.linalg.norm(st.get(1) - exact) <= TOL
    if H.is_hermitian:
        q.lanczos_evolve(H, st, 0, 2, 0.02, 33, 1)
        assert np.linalg.norm(st.get(1) - st.get(2)) <= TOL


def test_ground_state_at_the_limit(ctx, monkeypatch):
    """Real vectors, 95 columns (the most), 24,310 rows: 203 of 265 rows a block; against the passes over a
    basis in memory, as the persistent kernels' other tests bound it."""
    spec, ham = magnetised(17, 8)
    sec = q.Sector(spec.index, spec.constraints)
    out = []
    for split in (False, True):
        if split:
            monkeypatch.setenv("QD_KRYLOV_STEP", "split")
        H = sec.lower(ham)
        psi = q.getState(sec, 1)
        psi.set(0, q.start_vector(sec.dim, 5).astype(complex))
        s = q.Arnoldi.getSolver(sec, 95)
        n0 = ctx.launches()
        s.getGroundState(H, psi, 0)
        assert (ctx.launches() - n0 <= 4) != split
        out.append((s.eigenvalues(), psi.get(0)))
    (ea, pa), (eb, pb) = out
    assert len(ea) == len(eb) == 95
    assert np.allclose(ea, eb, rtol=0, atol=1e-11 * np.abs(eb).max())
    assert abs(abs(np.vdot(pa, pb)) - np.linalg.norm(pa) * np.linalg.norm(pb)) <= 1e-10
