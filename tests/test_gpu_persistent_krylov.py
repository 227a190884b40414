"""The persistent Krylov kernels against the kernels launched one by one (QD_KRYLOV_STEP=split) and the
dense or sparse propagator: one block and many, odd last slices, slices resident in shared memory and
streamed, real and complex operators, Hermitian and not, breakdown, incremental solves."""
import numpy as np
import pytest
import scipy.linalg as sl
import scipy.sparse.linalg as sla

import qudrip_gb300 as q
from qudrip_gb300 import _capi as A
from qudrip_gb300 import chains

pytestmark = pytest.mark.gpu

# Both forms hold the Krylov basis orthonormal to a few eps per vector and step; a step's result differs
# by at most m eps (1 + ||h H||) <= 33 * 2.2e-16 * 40, and three steps add up.
TOL = 1e-12


def flux_chain(L, phi=0.7):
    pre = q.getQbits(L)
    gc, ga, gz = q.getBoseGate(pre), q.getBoseGate(pre), q.getBoseGate(pre)
    gc << 0.5 * (q.pauli_x + q.II * q.pauli_y)
    ga << 0.5 * (q.pauli_x - q.II * q.pauli_y)
    gz << 0.5 * q.pauli_z
    t = 0.5 * np.exp(1j * phi / L)
    ham = q.getEmptyOperator()
    for i in range(L):
        j = (i + 1) % L
        ham = ham + t * (gc(i) * ga(j)) + np.conj(t) * (gc(j) * ga(i)) + 0.8 * (gz(i) * gz(j))
    return q.SectorSpec(pre, [q.getNset(pre) == L // 2]), ham


def damped_hubbard(L, nup, ndo, gamma=0.2):
    spec, ham = chains.hubbard_chain(L, nup, ndo, 4.0, -1.0)
    gate = q.getHopFermiGate(spec.index)
    for s in range(2 * L):
        ham = ham + (-0.5j * gamma) * gate(s, s)
    return spec, ham


def fields(L, seed=2):
    return chains.xxz_chain(L, 1.0, 0.7, True, np.random.default_rng(seed).uniform(-1, 1, L))


SYSTEMS = {
    "hubbard4_one_block": lambda: chains.hubbard_chain(4, 2, 2, 4.0, -1.0),  # 36 rows
    "damped5_many_blocks": lambda: damped_hubbard(5, 2, 3),                  # 100 rows, not Hermitian
    "xxz8_fields": lambda: fields(8),                                        # 70 rows: five blocks of 14
    "flux11": lambda: flux_chain(11),                                        # 462 rows, complex Hermitian
    "damped8": lambda: damped_hubbard(8, 4, 4),                              # 4,900 rows
    "flux17": lambda: flux_chain(17),                                        # 24,310 rows
    "xxz19_fields": lambda: fields(19),                                      # 92,378 rows: streamed
    "damped10_stream": lambda: damped_hubbard(10, 5, 5),                     # 63,504 rows
}


def objects(name):
    spec, ham = SYSTEMS[name]()
    sec = q.Sector(spec.index, spec.constraints)
    return sec, sec.lower(ham)


def evolve(sec, H, psi0, m, h, steps):
    st = q.getState(sec, steps + 1)
    st.set(0, psi0)
    s = q.Arnoldi.getSolver(sec, m)
    for t in range(steps):
        s.evolve(H, st(t), t, h)
    return [st.get(t + 1) for t in range(steps)], s.act_dim()


@pytest.mark.parametrize("name,m,h", [("hubbard4_one_block", 20, 0.05), ("damped5_many_blocks", 30, 0.1),
                                      ("xxz8_fields", 2, 0.05), ("xxz8_fields", 33, 0.05), ("flux11", 17, 0.2),
                                      ("damped8", 30, 0.01), ("flux17", 12, 0.05), ("xxz19_fields", 16, 0.05),
                                      ("damped10_stream", 33, 0.02), ("flux11", 33, 9.0)])
def test_evolve_matches_the_separate_kernels_and_the_propagator(ctx, monkeypatch, name, m, h):
    sec, H = objects(name)
    rng = np.random.default_rng(m)
    psi0 = rng.normal(size=sec.dim) + 1j * rng.normal(size=sec.dim)
    psi0 /= np.linalg.norm(psi0)
    got, act = evolve(sec, H, psi0, m, h, 3)
    monkeypatch.setenv("QD_KRYLOV_STEP", "split")
    ref, act_ref = evolve(sec, H, psi0, m, h, 3)
    monkeypatch.delenv("QD_KRYLOV_STEP")
    assert act == act_ref
    # a step far beyond the Krylov space's reach (h = 9) is compared as the same wrong answer
    for a, b in zip(got, ref):
        assert np.linalg.norm(a - b) <= (TOL if h < 1 else 1e-9)
    if m >= 12 and h < 1:
        exact = sla.expm_multiply(-1j * h * H.scipy().tocsc(), psi0)
        assert np.linalg.norm(got[0] - exact) <= 1e-8


def test_evolve_in_place_and_a_closed_space(ctx):
    sec, H = objects("hubbard4_one_block")
    w, v = np.linalg.eigh(H.scipy().toarray())
    x = v[:, 0] + 0.5 * v[:, 7] + 0.25j * v[:, 20]  # three levels: the space closes at the third step
    st = q.getState(sec, 1)
    st.set(0, x)
    s = q.Arnoldi.getSolver(sec, 20)
    s.evolve_inplace(H, st(0), 0, 0.3)
    assert s.act_dim() == 3
    ref = v @ (np.exp(-0.3j * w) * (v.conj().T @ (x / np.linalg.norm(x))))
    assert np.linalg.norm(st.get(0) - ref) <= TOL


@pytest.mark.parametrize("name,kdim,add,imag", [("xxz8_fields", 40, 7, False), ("flux11", 50, 20, False),
                                                ("xxz19_fields", 24, 11, False), ("xxz8_fields", 30, 30, True),
                                                ("hubbard4_one_block", 60, 9, False), ("damped8", 30, 13, True)])
def test_ground_state_calls_match_the_separate_kernels(ctx, monkeypatch, name, kdim, add, imag):
    sec, H = objects(name)
    v0 = q.start_vector(sec.dim, 5).astype(complex)
    if imag:
        v0 = v0 + 1j * q.start_vector(sec.dim, 6)
    out = []
    for form in ("one", "split"):
        if form == "split":
            monkeypatch.setenv("QD_KRYLOV_STEP", "split")
        sec, H = objects(name)
        psi = q.getState(sec, 1)
        psi.set(0, v0)
        s = q.Arnoldi.getSolver(sec, kdim)
        acts, evs = [], []
        while s.act_dim() < kdim:
            r = s.getGroundState(H, psi, 0, add)
            acts.append(s.act_dim())
            evs.append(s.eigenvalues().copy())
            if r.breakdown:
                break
        out.append((acts, evs, psi.get(0)))
    monkeypatch.delenv("QD_KRYLOV_STEP")
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1], out[1][1]):
        assert np.allclose(a, b, rtol=0, atol=1e-11 * np.abs(b).max())
    ov = abs(np.vdot(out[0][2], out[1][2])) / (np.linalg.norm(out[0][2]) * np.linalg.norm(out[1][2]))
    assert abs(ov - 1) <= 1e-10


def test_a_wait_that_runs_out_is_reported_and_the_next_step_is_unchanged(ctx, monkeypatch):
    """QD_STEP_WAIT_OUT keeps one block's sums back: every other block gives up after a few polls, the
    kernel ends, and the call reports a timeout; the next call carries the bits of one on a fresh operator."""
    sec, H = objects("flux11")
    psi0 = q.start_vector(sec.dim, 3).astype(complex)
    ref, _ = evolve(sec, H, psi0, 12, 0.05, 1)
    monkeypatch.setenv("QD_STEP_WAIT_OUT", "8")
    with pytest.raises(A.QDError) as e:
        evolve(sec, H, psi0, 12, 0.05, 1)
    assert e.value.code == A.QD_ERR_TIMEOUT
    monkeypatch.delenv("QD_STEP_WAIT_OUT")
    again, _ = evolve(sec, H, psi0, 12, 0.05, 1)
    sec2, H2 = objects("flux11")
    fresh, _ = evolve(sec2, H2, psi0, 12, 0.05, 1)
    assert np.array_equal(again[0], ref[0]) and np.array_equal(fresh[0], ref[0])


def bond_chain(L, seed=3):
    pre = q.getQbits(L)
    gc, ga, gz = q.getBoseGate(pre), q.getBoseGate(pre), q.getBoseGate(pre)
    gc << 0.5 * (q.pauli_x + q.II * q.pauli_y)
    ga << 0.5 * (q.pauli_x - q.II * q.pauli_y)
    gz << 0.5 * q.pauli_z
    J = np.random.default_rng(seed).uniform(0.3, 0.7, L)
    ham = q.getEmptyOperator()
    for i in range(L):
        j = (i + 1) % L
        ham = ham + float(J[i]) * (gc(i) * ga(j)) + float(J[i]) * (gc(j) * ga(i)) + 0.9 * (gz(i) * gz(j))
    return q.SectorSpec(pre, [q.getNset(pre) == L // 2]), ham


LANCZOS = {
    "uniform7_one_block": lambda: chains.xxz_chain(7, 1.0, 0.6, True, np.linspace(-1, 1, 7)),  # 35 rows
    "uniform8": lambda: fields(8),             # 70 rows: one cluster, a ragged last block
    "uniform13": lambda: chains.xy_chain(13),  # 1,716 rows
    "uniform18": lambda: fields(18),           # 48,620 rows: every cluster, several rows a thread
    "bonds9": lambda: bond_chain(9),
    "bonds15": lambda: bond_chain(15),
    "flux8": lambda: flux_chain(8),
    "flux16": lambda: flux_chain(16),
    "hubbard5_signs": lambda: chains.hubbard_chain(5, 2, 3, 4.0, -1.0, periodic=True),
}


def both_forms(monkeypatch, run):
    out = [run()]
    monkeypatch.setenv("QD_KRYLOV_STEP", "split")
    monkeypatch.setenv("QD_LANCZOS_STEP", "split")
    out.append(run())
    monkeypatch.delenv("QD_KRYLOV_STEP")
    monkeypatch.delenv("QD_LANCZOS_STEP")
    return out


@pytest.mark.parametrize("name,kdim,imag,mfree", [
    ("uniform7_one_block", 12, False, False), ("uniform8", 20, False, True), ("uniform13", 30, False, False),
    ("uniform18", 40, False, False), ("uniform13", 25, True, False), ("bonds9", 22, False, True),
    ("bonds15", 40, False, False), ("flux8", 18, False, False), ("flux16", 40, True, True),
    ("hubbard5_signs", 25, False, False), ("uniform8", 1, False, False)])
def test_lanczos_matches_the_separate_launches(ctx, monkeypatch, name, kdim, imag, mfree):
    """Krylov dimensions below the first spurious copy, where the recurrence is well-conditioned: the
    eigenvalues differ by a few eps ||H|| per step at most (40 steps, ||H|| <= 30 eigenvalue units: 1e-12)."""
    spec, ham = LANCZOS[name]()
    sec = q.Sector(spec.index, spec.constraints)
    v0 = q.start_vector(sec.dim, 8).astype(complex)
    if imag:
        v0 = v0 + 1j * q.start_vector(sec.dim, 9)

    def run():
        H = sec.lower(ham)
        psi = q.getState(sec, 1)
        psi.set(0, v0)
        s = q.LanczosSolver(sec, kdim, spmv=A.QD_SPMV_MATRIX_FREE if mfree else A.QD_SPMV_CSR)
        r = s.getGroundState(H, psi, 0)
        return r.act_dim, s.eigenvalues(), psi.get(0)

    a, b = both_forms(monkeypatch, run)
    assert a[0] == b[0]
    assert np.allclose(a[1], b[1], rtol=0, atol=1e-12 * np.abs(b[1]).max())
    assert abs(abs(np.vdot(a[2], b[2])) - np.linalg.norm(a[2]) * np.linalg.norm(b[2])) <= 1e-10


@pytest.mark.parametrize("name,m,h,steps", [("uniform7_one_block", 12, 0.2, 3), ("uniform8", 33, 0.3, 2),
                                            ("flux8", 2, 0.05, 3), ("bonds15", 24, 0.2, 4), ("flux16", 32, 0.25, 3),
                                            ("uniform18", 20, 0.1, 2), ("hubbard5_signs", 33, 2.5, 2)])
def test_short_exponential_matches_the_separate_launches(ctx, monkeypatch, name, m, h, steps):
    spec, ham = LANCZOS[name]()
    sec = q.Sector(spec.index, spec.constraints)
    H = sec.lower(ham)
    rng = np.random.default_rng(m)
    x = rng.normal(size=sec.dim) + 1j * rng.normal(size=sec.dim)
    x /= np.linalg.norm(x)

    def run():
        st = q.getState(sec, 2)
        st.set(0, x)
        act = q.lanczos_evolve(H, st, 0, 1, h, m, steps)
        return act, st.get(1), st.get(0)

    a, b = both_forms(monkeypatch, run)
    assert a[0] == b[0] and np.array_equal(a[2], x)
    assert np.linalg.norm(a[1] - b[1]) <= (TOL if h < 1 else 1e-9)
    if h * m < 10 and m > 12:
        exact = sla.expm_multiply(-1j * h * steps * H.scipy().tocsc(), x)
        assert np.linalg.norm(a[1] - exact) <= 1e-8


@pytest.mark.parametrize("name,kdim,imag", [("uniform8", 20, False), ("bonds15", 35, False), ("flux16", 35, True),
                                            ("hubbard5_signs", 25, True), ("uniform7_one_block", 10, False)])
def test_hermitian_lanczos_with_its_basis_kept_matches_two_passes(ctx, monkeypatch, name, kdim, imag):
    spec, ham = LANCZOS[name]()
    sec = q.Sector(spec.index, spec.constraints)
    H = sec.lower(ham)
    v0 = q.start_vector(sec.dim, 8).astype(complex)
    if imag:
        v0 = v0 + 1j * q.start_vector(sec.dim, 9)

    def run():
        psi = q.getState(sec, 1)
        psi.set(0, v0)
        s = q.Hermitian.LanczosSolver(sec, kdim)
        r = s.getGroundState(H, psi, 0)
        return (r.act_dim, r.breakdown, r.matvecs), s.eigenvalues(), psi.get(0), r.err

    a, b = both_forms(monkeypatch, run)
    assert a[0] == b[0]
    assert np.allclose(a[1], b[1], rtol=0, atol=1e-12 * np.abs(b[1]).max())
    assert abs(abs(np.vdot(a[2], b[2])) - np.linalg.norm(a[2]) * np.linalg.norm(b[2])) <= 1e-10
    assert abs(a[3] - b[3]) <= 1e-10
