"""The batched solver on start vectors that are not finite."""
import numpy as np
import pytest

import qudrip_gb300 as q
from qudrip_gb300 import chains

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_start_vector_that_is_not_finite_gives_nan_and_leaves_the_others_alone(ctx, bad):
    """dim 252 on one CTA, dim 12,870 on a cluster: eigenvalue and energy of the spoilt instances are NaN,
    the clean ones carry the bits of a call in which every instance is clean."""
    hams, v0s = [], []
    for L in (10, 16, 10, 16):
        spec, ham = chains.xxz_chain(L, 1.0, 1.0, True, np.random.default_rng(L).uniform(-1, 1, L))
        hams.append(q.Sector(spec.index, spec.constraints).lower(ham))
        v0s.append(q.start_vector(hams[-1].dim, L))
    ref = q.batch_lanczos(hams, v0s, 20)
    for i in (0, 1):
        v0s[i] = v0s[i].copy()
        v0s[i][7] = bad
    out = q.batch_lanczos(hams, v0s, 20)
    assert np.isnan(out[:2, :2]).all()
    assert np.array_equal(out[2:, :5], ref[2:, :5])
