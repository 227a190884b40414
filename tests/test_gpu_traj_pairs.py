"""Ensembles of more trajectories than CTAs in flight, which run two to a CTA: the same decisions and
observables as the FP64 form, for odd counts, one-warp sectors, signed entries, many jumps (both of a pair
in one step) and the workload's dimension.  Observables are complex64 sums: 2e-5, as for one to a CTA; a
decision differs when its random number is within 1e-6 of the rate, once in 100 runs of this file."""
import numpy as np
import pytest

import qudrip_gb300 as q
from qudrip_gb300 import chains

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,nup,ndo,periodic,gamma,dt,steps,ntraj", [
    (2, 1, 1, False, 3.0, 0.1, 20, 5001),    # dim 4
    (4, 2, 2, False, 2.0, 0.05, 20, 5001),   # dim 36, one warp
    (4, 2, 2, True, 8.0, 0.05, 20, 5000),    # entries of both signs, jumps in most steps
    (6, 3, 3, True, 1.0, 0.05, 6, 1301),     # dim 400
    (8, 4, 4, False, 1.0, 0.01, 4, 155),     # dim 4,900, one CTA an SM
])
def test_pairs_equal_the_fp64_form(ctx, monkeypatch, L, nup, ndo, periodic, gamma, dt, steps, ntraj):
    spec, ham = chains.hubbard_chain(L, nup, ndo, 4.0, -1.0, periodic=periodic)
    g = q.getHopFermiGate(spec.index)
    for s in range(2 * L):
        ham = ham + (-0.5j * gamma) * g(s, s)
    sec = q.Sector(spec.index, spec.constraints)
    H = sec.lower(ham)
    rng = np.random.default_rng(L)
    psi0 = rng.normal(size=sec.dim) + 1j * rng.normal(size=sec.dim)
    args = (ntraj, steps, dt, gamma, 11, min(16, sec.dim + 1), list(range(2 * L)), [(i, i + L) for i in range(L)])
    mean, err, st = q.traj_run(H, psi0, *args)
    assert st.path == 0
    monkeypatch.setenv("QD_TRAJ_ARNOLDI", "1")
    mean64, err64, st64 = q.traj_run(H, psi0, *args)
    assert st64.path == 1
    assert st.jumps == st64.jumps and st.jumps > 0
    assert np.abs(mean - mean64).max() < 2e-5
    assert np.abs(err - err64).max() < 2e-5
