"""What operators and contexts keep between calls: plans, buffers, and the idle memory of a context."""
import numpy as np
import pytest

import qudrip_gb300 as q
from qudrip_gb300 import chains

from test_gpu_persistent_krylov import flux_chain

pytestmark = pytest.mark.gpu


def test_a_sector_too_large_for_the_persistent_form_is_looked_at_once(ctx, monkeypatch):
    """Complex vectors of 705,432 rows do not fit one block per SM: after the first call, which finds that
    out, a call launches what it launches step by step."""
    spec, ham = flux_chain(22)
    sec = q.Sector(spec.index, spec.constraints)
    psi = q.getState(sec, 2)
    psi.set(0, q.start_vector(sec.dim, 1).astype(complex))
    count = {}
    for split in (False, True):
        if split:
            monkeypatch.setenv("QD_KRYLOV_STEP", "split")
        H = sec.lower(ham)
        for _ in range(3):
            n0 = ctx.launches()
            q.lanczos_evolve(H, psi, 0, 1, 0.05, 4, 1)
            count[split] = ctx.launches() - n0
    assert count[False] == count[True]
