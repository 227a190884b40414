"""lanczos_evolve over times far beyond the norm of the operator, on Krylov spaces that close, so that the
result is known whatever the time."""
import numpy as np
import pytest

import qudrip_gb300 as q
from qudrip_gb300 import chains

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("system,rows", [("one_block", 36), ("many_blocks", 252)])
@pytest.mark.parametrize("theta", [3e2, 2e3, 3e6])
def test_a_long_step_on_a_closed_space(ctx, system, rows, theta):
    """Three levels of H: the space closes at the third step.  Both sides know the levels to rows eps ||H||
    at worst, so their phases agree to 2 rows eps theta; the scaled and squared exponential adds its
    m 2^s eps <= 33 eps theta."""
    if system == "one_block":
        spec, ham = chains.hubbard_chain(4, 2, 2, 4.0, -1.0)
    else:
        spec, ham = chains.xxz_chain(10, 1.0, 0.7, True, np.linspace(-1, 1, 10))
    sec = q.Sector(spec.index, spec.constraints)
    assert sec.dim == rows
    H = sec.lower(ham)
    w, v = np.linalg.eigh(H.scipy().toarray())
    x = v[:, 0] + 0.5 * v[:, 7] + 0.25j * v[:, 20]
    x /= np.linalg.norm(x)
    h = theta / np.abs(w).max()
    st = q.getState(sec, 2)
    st.set(0, x)
    act = q.lanczos_evolve(H, st, 0, 1, h, 20, 2)
    assert act == 3
    ref = v @ (np.exp(-2j * h * w) * (v.conj().T @ x))
    assert np.linalg.norm(st.get(1) - ref) <= 2 * (2 * rows + 33) * 2.3e-16 * theta


@pytest.mark.parametrize("h", [np.nan, np.inf])
def test_a_step_that_is_not_finite_gives_nan(ctx, h):
    spec, ham = chains.xxz_chain(10, 1.0, 0.7, True, np.linspace(-1, 1, 10))
    sec = q.Sector(spec.index, spec.constraints)
    H = sec.lower(ham)
    st = q.getState(sec, 2)
    st.set(0, q.start_vector(sec.dim, 1).astype(complex))
    q.lanczos_evolve(H, st, 0, 1, h, 12, 1)
    assert np.isnan(st.get(1)).all()
