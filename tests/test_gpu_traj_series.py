"""The series of a trajectory step: Chebyshev's where H_eff - mu is Hermitian (one damping on the whole sector,
or none), Taylor's where it is not, against the FP64 form at small and large steps (one and several sub-steps).
Observables are complex64 sums and a step's series is cut at 1e-8: 2e-5, as for the form as a whole."""
import numpy as np
import pytest

import qudrip_gb300 as q
from qudrip_gb300 import chains

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [0.0004, 0.01, 0.04, 0.3])
@pytest.mark.parametrize("damping", ["none", "uniform", "half", "complex_hop"])
def test_series_equals_the_fp64_form(ctx, monkeypatch, dt, damping):
    L = 5
    spec, ham = chains.hubbard_chain(L, 3, 2, 4.0, -1.0)
    g = q.getHopFermiGate(spec.index)
    chan = list(range(2 * L)) if damping != "half" else [0, 3, 6]
    gamma = 0.0 if damping == "none" else 0.4
    for s in chan:
        ham = ham + (-0.5j * gamma) * g(s, s)
    if damping == "complex_hop":  # every off-diagonal value -1 + 0.3i: neither real nor Hermitian
        for i in range(L - 1):
            for o in (0, L):
                ham = ham + 0.3j * (g(i + 1 + o, i + o) + g(i + o, i + 1 + o))
    sec = q.Sector(spec.index, spec.constraints)
    H = sec.lower(ham)
    rng = np.random.default_rng(7)
    psi0 = rng.normal(size=sec.dim) + 1j * rng.normal(size=sec.dim)
    args = (40, 25, dt, gamma, 5, 32, chan, [(i, i + L) for i in range(L)])
    mean, err, st = q.traj_run(H, psi0, *args)
    assert st.path == 0
    monkeypatch.setenv("QD_TRAJ_ARNOLDI", "1")
    mean64, err64, st64 = q.traj_run(H, psi0, *args)
    assert st64.path == 1
    assert st.jumps == st64.jumps
    assert np.abs(mean - mean64).max() < 2e-5
