"""Observable lists in one launch per 32 operators (qd_obs_eval) against host products."""
import numpy as np
import pytest

import qudrip_gb300 as q
from qudrip_gb300 import chains

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 33])
@pytest.mark.parametrize("L,nup,ndo", [(3, 1, 2), (6, 3, 3), (8, 4, 3)])
def test_observables_in_one_launch(ctx, L, nup, ndo, count):
    """One launch per 32 operators: batches of one operator and of 33, real and complex, diagonal and not."""
    spec, ham = chains.hubbard_chain(L, nup, ndo, 4.0, -1.0)
    sec = q.Sector(spec.index, spec.constraints)
    g = q.getHopFermiGate(spec.index)
    ops = []
    for i in range(count):
        a, b = i % L, (i + 1) % L
        ops.append([1.0 * g(a, a), 1j * g(a, b) - 1j * g(b, a), 0.5 * g(a + L, b + L) + 0.5 * g(b + L, a + L)][i % 3])
    mats = [sec.lower(o) for o in ops]
    x = np.random.default_rng(L).normal(size=sec.dim) + 1j * np.random.default_rng(L + 1).normal(size=sec.dim)
    st = q.getState(sec, 1)
    st.set(0, x)
    got = q.obs_eval(st, 0, mats)
    for e, M in zip(got, mats):
        Ms = M.scipy()
        # an FP64 sum of dim terms over threads and blocks: a few eps of the sum of magnitudes
        assert abs(e - np.vdot(x, Ms @ x)) <= 1e-14 * max(1.0, np.abs(np.conj(x) * (Ms @ x)).sum())
    assert np.array_equal(got, q.obs_eval(st, 0, mats))
