"""Krylov steps from a state on one basis row: its amplitudes fall by orders of magnitude with every hop, and
each keeps its own relative accuracy, far below the rounding of the largest."""
import numpy as np
import pytest

import qudrip_gb300 as q
from qudrip_gb300 import chains

from test_gpu_persistent_krylov import damped_hubbard, flux_chain

pytestmark = pytest.mark.gpu

STEPS, M = 3, 20

SYSTEMS = {
    "xxz12": (lambda: chains.xxz_chain(12, 1.0, 0.7, True, np.linspace(-1, 1, 12)), 4e-3),
    "flux11": (lambda: flux_chain(11), 4e-3),                          # complex
    "damped6": (lambda: damped_hubbard(6, 3, 3), 2e-3),                # not Hermitian
    "xxz16": (lambda: chains.xxz_chain(16, 1.0, 0.7, True), 4e-3),     # 12,870 rows
}


def taylor(Hs, x, t):
    """exp(-i t H) x: every amplitude's leading term is its first, so each is accurate by itself."""
    out, term = x.copy(), x.copy()
    for p in range(1, 40):
        term = (-1j * t / p) * (Hs @ term)
        out = out + term
    return out


@pytest.mark.parametrize("name", sorted(SYSTEMS))
@pytest.mark.parametrize("form", ["one", "split"])
def test_small_amplitudes_keep_their_accuracy(ctx, monkeypatch, name, form):
    """Rows up to eight hops away (amplitudes down to some 1e-24), three steps of a Krylov space of 20: its
    truncation is below 1e-10 of each (||h H||^12), and some hundred roundings of 1e-16 amplified by the
    ratio of neighbouring shells (1e3 at most) stay below 1e-9."""
    if form == "split":
        monkeypatch.setenv("QD_KRYLOV_STEP", "split")
    make, h = SYSTEMS[name]
    spec, ham = make()
    sec = q.Sector(spec.index, spec.constraints)
    H = sec.lower(ham)
    Hs = H.scipy().tocsr()
    x = np.zeros(sec.dim, dtype=complex)
    x[0] = 1.0
    reach = x != 0
    for _ in range(8):
        reach = reach | ((abs(Hs) @ reach.astype(float)) > 0)
    st = q.getState(sec, STEPS + 1)
    st.set(0, x)
    s = q.Arnoldi.getSolver(sec, M)
    ref = x
    for t in range(STEPS):
        s.evolve(H, st(t), t, h)
        ref = taylor(Hs, ref, h)
    got = st.get(STEPS)
    if not H.is_hermitian:
        ref, got = ref / np.linalg.norm(ref), got / np.linalg.norm(got)
    err = np.abs(got - ref)[reach] / np.abs(ref)[reach]
    assert np.abs(ref)[reach].min() < 1e-18
    assert err.max() <= 1e-9
