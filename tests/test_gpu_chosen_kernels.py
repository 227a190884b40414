"""Product kernels chosen with qd_ham_set_spmv_kernel are launched by every call that forms products on the
stored matrix, also where it has a faster product of its own otherwise."""
import ctypes as C

import numpy as np
import pytest

import qudrip_gb300 as q
from qudrip_gb300 import _capi as A
from qudrip_gb300 import chains

from test_gpu_persistent_krylov import bond_chain, flux_chain

pytestmark = pytest.mark.gpu

SYSTEMS = {
    "uniform12": lambda: chains.xxz_chain(12, 1.0, 0.7, True, np.linspace(-1, 1, 12)),
    "bonds12": lambda: bond_chain(12),
    "flux11": lambda: flux_chain(11),
}


def ground(sec, H, psi):
    q.LanczosSolver(sec, 15).getGroundState(H, psi, 0)


def arnoldi(sec, H, psi):
    s = q.Arnoldi.getSolver(sec, 15)
    s.getGroundState(H, psi, 0, 8)
    s.getGroundState(H, psi, 0, 7)


CALLS = {  # the call and its products
    "ground": (ground, 15),
    "hermitian": (lambda sec, H, psi: q.Hermitian.LanczosSolver(sec, 15).getGroundState(H, psi, 0), 31),
    "arnoldi": (arnoldi, 15),
    "evolve": (lambda sec, H, psi: q.Arnoldi.getSolver(sec, 15).evolve_inplace(H, psi, 0, 0.1), 14),
}


@pytest.mark.parametrize("name", sorted(SYSTEMS))
@pytest.mark.parametrize("call", sorted(CALLS))
def test_a_chosen_kernel_is_launched_for_every_product(ctx, monkeypatch, name, call):
    spec, ham = SYSTEMS[name]()
    sec = q.Sector(spec.index, spec.constraints)
    x = q.start_vector(sec.dim, 3).astype(complex)
    fn, products = CALLS[call]
    out = {}
    for kernel, split in ((None, False), (101, False), (101, True), (111, False)):
        if split:  # the form that always launched it
            monkeypatch.setenv("QD_KRYLOV_STEP", "split")
            monkeypatch.setenv("QD_LANCZOS_STEP", "split")
        H = sec.lower(ham)
        if kernel:
            A.call("qd_ham_set_spmv_kernel", H.handle, kernel)
        psi = q.getState(sec, 1)
        psi.set(0, x)
        n0 = ctx.launches()
        fn(sec, H, psi)
        out[kernel, split] = psi.get(0)
        if kernel:
            assert ctx.launches() - n0 >= products
        monkeypatch.undo()
    assert np.array_equal(out[101, False], out[101, True])
    for key in ((101, False), (111, False)):
        a, b = out[key], out[None, False]
        assert abs(abs(np.vdot(a, b)) - np.linalg.norm(a) * np.linalg.norm(b)) <= 1e-10


def test_an_operator_list_launches_its_chosen_kernels(ctx):
    spec, ham = SYSTEMS["bonds12"]()
    sec = q.Sector(spec.index, spec.constraints)
    psi = q.getState(sec, 1)
    psi.set(0, q.start_vector(sec.dim, 3) + 1j * q.start_vector(sec.dim, 4))
    ops = [sec.lower(ham) for _ in range(40)]
    n0 = ctx.launches()
    ref = q.obs_eval(psi, 0, ops)
    assert ctx.launches() - n0 == 2  # 32 a launch
    for i in (0, 5, 33):
        A.call("qd_ham_set_spmv_kernel", ops[i].handle, 101 + i % 4)
    n0 = ctx.launches()
    got = q.obs_eval(psi, 0, ops)
    assert ctx.launches() - n0 == 2 + 3
    assert np.max(np.abs(got - ref)) <= 1e-13 * abs(ref[0])


def test_the_autotuner_keeps_the_faster_form(ctx):
    """It times products launched one by one, so its choice does not take an operator off the form that
    launches none."""
    spec, ham = SYSTEMS["bonds12"]()
    sec = q.Sector(spec.index, spec.constraints)
    H, H2 = sec.lower(ham), sec.lower(ham)
    chosen, ms = C.c_int(), C.c_double()
    A.call("qd_ham_autotune", H2.handle, 2, C.byref(chosen), C.byref(ms))
    out = []
    for op in (H, H2):
        psi = q.getState(sec, 1)
        psi.set(0, q.start_vector(sec.dim, 3).astype(complex))
        ground(sec, op, psi)
        out.append(psi.get(0))
    assert np.array_equal(*out)


@pytest.mark.parametrize("call", ["ground", "short", "evolve"])
def test_a_later_choice_replaces_what_a_graph_launches(ctx, call):
    """Recurrences are captured once and replayed; another choice on the same operator gives the bits of that
    kernel on a fresh one (104 adds a row's entries over eight lanes, 110 in their order)."""
    spec, ham = SYSTEMS["bonds12"]()
    sec = q.Sector(spec.index, spec.constraints)
    fn = {"ground": ground,
          "short": lambda sec, H, psi: q.lanczos_evolve(H, psi, 0, 0, 0.1, 12, 2),
          "evolve": CALLS["evolve"][0]}[call]
    psi = q.getState(sec, 1)

    def run(H, kernel):
        A.call("qd_ham_set_spmv_kernel", H.handle, kernel)
        for _ in range(3):  # the first runs may not be captured yet
            psi.set(0, q.start_vector(sec.dim, 3).astype(complex))
            fn(sec, H, psi)
        return psi.get(0)

    H = sec.lower(ham)
    first = run(H, 110)
    second = run(H, 104)
    assert not np.array_equal(first, second)
    assert np.array_equal(second, run(sec.lower(ham), 104))
    assert np.array_equal(first, run(H, 110))
