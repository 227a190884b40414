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


def lowest(sec, H, kdim, add=-1):
    psi = q.getState(sec, 1)
    psi.set(0, q.start_vector(sec.dim, 3).astype(complex))
    s = q.LanczosSolver(sec, kdim)
    while s.act_dim() < kdim:
        s.getGroundState(H, psi, 0, add)
    return s.eigenvalues(), psi.get(0)


def test_long_uniform_solves_run_in_pieces_with_the_same_bits(ctx):
    """48,620 rows: the fixed-point copies of 171 steps are the limit of one launch.  One call (two pieces), a
    call a few steps short of the limit and grown over it, and pieces of the caller's."""
    spec, ham = chains.xxz_chain(18, 1.0, 0.7, True)
    sec = q.Sector(spec.index, spec.constraints)
    H = sec.lower(ham)
    n0 = ctx.launches()
    ref = lowest(sec, H, 180)
    assert ctx.launches() - n0 < 20
    for add in (165, 60):
        got = lowest(sec, sec.lower(ham), 180, add)
        assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])


def used():
    torch = pytest.importorskip("torch")
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_an_operator_keeps_no_basis_after_a_solve(ctx):
    """Memory that 24 operators hold beyond their matrices after a Hermitian and a uniform Lanczos solve:
    the basis of the open solve (a later call may grow it), not the Hermitian solver's or the copies."""
    spec, ham = chains.xxz_chain(18, 1.0, 0.7, True)
    sec = q.Sector(spec.index, spec.constraints)
    c = q.Context()
    sec = q.Sector(spec.index, spec.constraints, ctx=c)
    hams = [sec.lower(ham) for _ in range(24)]
    vec = sec.dim * 8
    psi = q.getState(sec, 1)

    def solve(H):
        psi.set(0, q.start_vector(sec.dim, 3).astype(complex))
        q.Hermitian.LanczosSolver(sec, 60).getGroundState(H, psi, 0)
        psi.set(0, q.start_vector(sec.dim, 3).astype(complex))
        q.LanczosSolver(sec, 60).getGroundState(H, psi, 0)

    solve(hams[0])  # the shared buffers
    u0 = used()
    for H in hams[1:]:
        solve(H)
    # 61 vectors of the open solve and some thirty of workspace an operator; the Hermitian basis would add 62
    # and the copies 122
    assert (used() - u0) / 23 < 110 * vec


def test_idle_memory_of_one_context_serves_another(ctx):
    """A context keeps freed buffers (two 22-site operators': some 600 MB); when the device is full but for
    150 MB, another context's state of 400 MB takes their place."""
    torch = pytest.importorskip("torch")
    spec, ham = chains.xxz_chain(22, 1.0, 0.7, True, np.linspace(-1, 1, 22))
    a, b = q.Context(), q.Context()
    sec = q.Sector(spec.index, spec.constraints, ctx=a)
    for H in [sec.lower(ham), sec.lower(ham)]:
        H.close()
    small, _ = chains.xy_chain(20)  # 184,756 rows: 2.96 MB a column
    other = q.Sector(small.index, small.constraints, ctx=b)
    free, _ = torch.cuda.mem_get_info()
    block = torch.empty(free - (150 << 20), dtype=torch.uint8, device="cuda")
    try:
        st = q.getState(other, 135)
        st.close()
    finally:
        del block
        torch.cuda.empty_cache()
