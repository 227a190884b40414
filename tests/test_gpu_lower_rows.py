"""Row-wise lowering by flip groups against the oracle, bit for bit: rings whose closing bond shares its
highest bit with another bond (columns out of group order), several flips per highest bit, several terms
on one flip, Jordan-Wigner signs, diagonal-only and empty operators, loose sectors (ranks by search), rows
longer than 64 entries, and operators too many for the staged tables."""
import numpy as np
import pytest

import oracle as O
import qudrip_gb300 as q
from qudrip_gb300 import chains

pytestmark = pytest.mark.gpu


def ladders(L):
    pre = q.getQbits(L)
    gc, ga, gz = q.getBoseGate(pre), q.getBoseGate(pre), q.getBoseGate(pre)
    gc << 0.5 * (q.pauli_x + q.II * q.pauli_y)
    ga << 0.5 * (q.pauli_x - q.II * q.pauli_y)
    gz << 0.5 * q.pauli_z
    return pre, gc, ga, gz


def all_pairs(L, n, tight=0, repeat=1):
    pre, gc, ga, gz = ladders(L)
    ham = q.getEmptyOperator()
    for k in range(repeat):
        for i in range(L):
            for j in range(L):
                if i != j:
                    ham = ham + (0.1 * (i + 1) + 0.01 * j + 0.3j * k) * (gc(i) * ga(j))
            ham = ham + (0.2 + k) * gz(i)
    return q.SectorSpec(pre, [q.getNset(pre) == n], tight), ham


def diagonal_only(L):
    pre, _, _, gz = ladders(L)
    ham = q.getEmptyOperator()
    for i in range(L - 1):
        ham = ham + 0.7 * (gz(i) * gz(i + 1)) + (-0.7) * (gz(i) * gz(i + 1))
    return q.SectorSpec(pre, [q.getNset(pre) == L // 2]), ham


CASES = {
    "ring3": lambda: chains.xxz_chain(3, 1.0, 0.7, True),
    "ring11_fields": lambda: chains.xxz_chain(11, 1.0, 0.7, True, np.linspace(-1, 1, 11)),
    "all_pairs8": lambda: all_pairs(8, 4),
    "all_pairs8_twice": lambda: all_pairs(8, 3, repeat=2),      # two terms per flip
    "all_pairs7_loose": lambda: all_pairs(7, 3, tight=1),       # sector without product structure
    "all_pairs18_rows_of_82": lambda: all_pairs(18, 9),         # more than 64 entries a row, tables past 44 KB
    "fermions_periodic": lambda: chains.hubbard_chain(5, 2, 3, 4.0, -1.0, periodic=True),
    "diagonal_cancels": lambda: diagonal_only(9),
    "empty": lambda: (diagonal_only(6)[0], q.getEmptyOperator()),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_rows_equal_the_oracle_bit_for_bit(ctx, name):
    spec, ham = CASES[name]()
    H = q.Sector(spec.index, spec.constraints, spec.tight).lower(ham)
    o = O.Ham(O.Sector(spec), ham)
    assert (H.dim, H.nnz) == (o.dim, o.nnz)
    M = o.scipy().tocsr()
    M.sort_indices()
    rp, ci, v = H.csr()
    assert np.array_equal(rp, M.indptr) and np.array_equal(ci, M.indices) and np.array_equal(v, M.data)
    assert H.max_row_nnz == (int(np.diff(M.indptr).max()) if o.nnz else 0)
    assert H.is_real == (not np.any(M.data.imag != 0))
    assert H.is_hermitian == (abs(M - M.getH()).max() <= 1e-12 if o.nnz else True)
