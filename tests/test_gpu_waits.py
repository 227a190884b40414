"""The bounded waits of the persistent Krylov kernels.  QD_STEP_WAIT_OUT holds one block's rows and sums back
and lets every other block give up after a few polls: the kernel ends, the call reports a timeout and leaves
the caller's state as it was, and the next call carries the bits of one on a fresh operator."""
import numpy as np
import pytest

import qudrip_gb300 as q
from qudrip_gb300 import _capi as A
from qudrip_gb300 import chains

from test_gpu_persistent_krylov import bond_chain, flux_chain

pytestmark = pytest.mark.gpu

SYSTEMS = {
    "uniform10": lambda: chains.xxz_chain(10, 1.0, 0.7, True, np.linspace(-1, 1, 10)),
    "bonds10": lambda: bond_chain(10),
    "flux11": lambda: flux_chain(11),
}


def lanczos(spmv):
    def run(sec, H, psi):
        q.LanczosSolver(sec, 15, spmv=spmv).getGroundState(H, psi, 0)
    return run


def grown(sec, H, psi):
    s = q.Arnoldi.getSolver(sec, 20)
    s.getGroundState(H, psi, 0, 8)
    s.getGroundState(H, psi, 0, 8)


CALLS = {
    "lanczos": lanczos(A.QD_SPMV_CSR),
    "lanczos_mfree": lanczos(A.QD_SPMV_MATRIX_FREE),
    "hermitian": lambda sec, H, psi: q.Hermitian.LanczosSolver(sec, 15).getGroundState(H, psi, 0),
    "arnoldi": grown,
    "evolve_in_place": lambda sec, H, psi: q.Arnoldi.getSolver(sec, 12).evolve_inplace(H, psi, 0, 0.1),
    "evolve": lambda sec, H, psi: q.Arnoldi.getSolver(sec, 12).evolve(H, psi, 0, 0.1),
    "short_in_place": lambda sec, H, psi: q.lanczos_evolve(H, psi, 0, 0, 0.1, 12, 3),
    "short": lambda sec, H, psi: q.lanczos_evolve(H, psi, 0, 1, 0.1, 12, 1),
    "short_long_time": lambda sec, H, psi: q.lanczos_evolve(H, psi, 0, 0, 100.0, 12, 1),
}


# the FP64 matrix-free product has no kernel that waits
@pytest.mark.parametrize("name,call", [(n, c) for n in SYSTEMS for c in CALLS
                                       if c != "lanczos_mfree" or n == "uniform10"])
def test_a_wait_that_runs_out_leaves_the_state_alone(ctx, monkeypatch, name, call):
    spec, ham = SYSTEMS[name]()
    sec = q.Sector(spec.index, spec.constraints)
    x = q.start_vector(sec.dim, 3).astype(complex)
    H = sec.lower(ham)
    psi = q.getState(sec, 2)

    def fill():
        psi.set(0, x)
        psi.set(1, 2.0 * x)

    fill()
    CALLS[call](sec, H, psi)
    ref = [psi.get(0), psi.get(1)]
    fill()
    monkeypatch.setenv("QD_STEP_WAIT_OUT", "8")
    with pytest.raises(A.QDError) as e:
        CALLS[call](sec, H, psi)
    assert e.value.code == A.QD_ERR_TIMEOUT
    monkeypatch.delenv("QD_STEP_WAIT_OUT")
    assert np.array_equal(psi.get(0), x) and np.array_equal(psi.get(1), 2.0 * x)
    for op in (H, sec.lower(ham)):
        fill()
        CALLS[call](sec, op, psi)
        assert np.array_equal(psi.get(0), ref[0]) and np.array_equal(psi.get(1), ref[1])
