"""The tests of the Lanczos step's kernels on sectors that solves run in one launch for all steps: here each
step is launched by itself (QD_KRYLOV_STEP=split), so the kernels that these tests name are the ones that run."""
import numpy as np
import pytest

import qudrip_gb300 as q
from qudrip_gb300 import _capi as A
from qudrip_gb300 import chains

from test_gpu_edges import (  # noqa: F401
    test_step_barrier_wait_runs_out_and_next_solve_is_unchanged,
    test_step_mailbox_across_runs_and_forms,
)
from test_gpu_fx import (  # noqa: F401
    test_block_layout_step_matches_stored_columns,
    test_columns_on_the_fly_bit_identical_to_stored_columns,
    test_one_launch_step_matches_two_launch_step,
)
from test_gpu_mfree import (  # noqa: F401
    test_matrix_free_nonuniform_keeps_fp64_product,
    test_matrix_free_uniform_form_bit_identical_to_csr,
)

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def launched(monkeypatch):
    monkeypatch.setenv("QD_KRYLOV_STEP", "split")


@pytest.mark.parametrize("kernel", [A.QD_SPMV_FX, A.QD_SPMV_FX_SLOTS, A.QD_SPMV_FX_BLOCK, "staged", "mfree"])
def test_a_solve_launches_its_steps(ctx, monkeypatch, kernel):
    spec, ham = chains.xxz_chain(12, 1.0, 0.7, True)
    sec = q.Sector(spec.index, spec.constraints)
    if kernel == "staged":
        monkeypatch.setenv("QD_FX_BLOCK_STAGED", "1")
    H = sec.lower(ham)
    if kernel != "mfree":
        A.call("qd_ham_set_spmv_kernel", H.handle, A.QD_SPMV_FX_BLOCK if kernel == "staged" else kernel)
    psi = q.getState(sec, 1)
    psi.set(0, q.start_vector(sec.dim, 3).astype(complex))
    n0 = ctx.launches()
    q.LanczosSolver(sec, 30, spmv=A.QD_SPMV_MATRIX_FREE if kernel == "mfree" else A.QD_SPMV_CSR) \
        .getGroundState(H, psi, 0)
    assert ctx.launches() - n0 >= 30
    assert np.isfinite(psi.get(0)).all()
