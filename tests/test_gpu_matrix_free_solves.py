"""Matrix-free Lanczos solves in the persistent recurrence: columns and values from the compiled transitions,
in their order, against the stored matrix and the kernels launched one by one."""
import numpy as np
import pytest

import qudrip_gb300 as q
from qudrip_gb300 import _capi as A
from qudrip_gb300 import chains

from test_gpu_fx import two_species_xy
from test_gpu_persistent_krylov import bond_chain, flux_chain

pytestmark = pytest.mark.gpu


def loose(spec, ham):
    return q.SectorSpec(spec.index, spec.constraints, tight=1), ham  # ranked by search, not by tables


NONUNIFORM = {
    "bonds6_one_block": lambda: bond_chain(6),       # 20 rows
    "bonds9": lambda: bond_chain(9),                 # 126 rows: a row shared by four threads
    "bonds15": lambda: bond_chain(15),               # 6,435 rows
    "bonds18": lambda: bond_chain(18),               # 48,620 rows: rows in order of their length
    "bonds12_loose": lambda: loose(*bond_chain(12)),
    "flux12": lambda: flux_chain(12),
    "hubbard5_signs": lambda: chains.hubbard_chain(5, 2, 3, 4.0, -1.0, periodic=True),
}
UNIFORM = {
    "xxz8_one_cluster": lambda: chains.xxz_chain(8, 1.0, 0.7, True, np.linspace(-1, 1, 8)),
    "xxz18": lambda: chains.xxz_chain(18, 1.0, 0.7, True),
    "xy13_open": lambda: chains.xy_chain(13),
    "two_species": lambda: two_species_xy(6, True),
}


def solve(sec, H, v0, kdim, spmv, add=-1):
    psi = q.getState(sec, 1)
    psi.set(0, v0)
    s = q.LanczosSolver(sec, kdim, spmv=spmv)
    while s.act_dim() < kdim:
        s.getGroundState(H, psi, 0, add)
    return s.eigenvalues(), psi.get(0)


@pytest.mark.parametrize("name", sorted(NONUNIFORM))
@pytest.mark.parametrize("add", [-1, 7])
def test_the_fp64_product_reads_the_transitions(ctx, monkeypatch, name, add):
    """A row's entries are summed in another order than the stored matrix's, so the bits differ from a
    solve on the matrix; both, and the launches one by one, agree to a few eps ||H|| per step."""
    spec, ham = NONUNIFORM[name]()
    sec = q.Sector(spec.index, spec.constraints, spec.tight)
    H = sec.lower(ham)
    v0 = q.start_vector(sec.dim, 8).astype(complex)
    kdim = min(24, sec.dim // 2)
    ev, psi = solve(sec, H, v0, kdim, A.QD_SPMV_MATRIX_FREE, add)
    ev_csr, psi_csr = solve(sec, H, v0, kdim, A.QD_SPMV_CSR, add)
    monkeypatch.setenv("QD_KRYLOV_STEP", "split")
    monkeypatch.setenv("QD_LANCZOS_STEP", "split")
    ev_one, psi_one = solve(sec, sec.lower(ham), v0, kdim, A.QD_SPMV_MATRIX_FREE, add)
    monkeypatch.undo()
    assert not np.array_equal(psi, psi_csr)
    for e, p in ((ev_csr, psi_csr), (ev_one, psi_one)):
        assert np.allclose(ev, e, rtol=0, atol=1e-12 * np.abs(e).max())
        assert abs(abs(np.vdot(psi, p)) - np.linalg.norm(psi) * np.linalg.norm(p)) <= 1e-10


@pytest.mark.parametrize("name", sorted(UNIFORM))
def test_uniform_couplings_carry_the_same_bits_from_every_source_of_columns(ctx, name):
    spec, ham = UNIFORM[name]()
    sec = q.Sector(spec.index, spec.constraints)
    v0 = q.start_vector(sec.dim, 8).astype(complex)
    H = sec.lower(ham)
    ref = solve(sec, H, v0, 24, A.QD_SPMV_CSR)
    got = [solve(sec, H, v0, 24, A.QD_SPMV_MATRIX_FREE)]
    for kernel in (A.QD_SPMV_FX_SLOTS, A.QD_SPMV_FX_BLOCK, A.QD_SPMV_FX):
        A.call("qd_ham_set_spmv_kernel", H.handle, kernel)
        got.append(solve(sec, H, v0, 24, A.QD_SPMV_CSR))
    for ev, psi in got:
        assert np.array_equal(ev, ref[0]) and np.array_equal(psi, ref[1])


@pytest.mark.parametrize("make", [lambda: chains.xy_chain(9), lambda: two_species_xy(4, False)])
def test_targets_outside_the_sector_are_dropped(ctx, make):
    """Terms that raise two sites leave the sector from every state they apply to."""
    spec, ham = make()
    gp = q.getBoseGate(spec.index)
    gp << 0.5 * (q.pauli_x + q.II * q.pauli_y)
    for i in range(spec.index.nbits - 1):
        ham = ham + 0.3 * (gp(i) * gp(i + 1))
    sec = q.Sector(spec.index, spec.constraints)
    H = sec.lower(ham)
    st = q.getState(sec, 2)
    x = q.start_vector(sec.dim, 2) + 1j * q.start_vector(sec.dim, 3)
    st.set(0, x)
    q.apply(H, st, 0, st, 1, matrix_free=True)
    ref = H.scipy() @ x
    assert np.max(np.abs(st.get(1) - ref)) <= 1e-14 * np.abs(H.scipy()).sum(axis=1).max() * np.abs(x).max()
