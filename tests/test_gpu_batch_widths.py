"""The batched solver's cluster sizes, which follow the work of a call: every size on uneven row slices, few and
many steps (down to one: a 1 x 1 tridiagonal matrix), exhausted spaces, each against the lowest value of the same
Krylov space in FP64.  FP32 products with FP64 refinement: the refined energy is within 1e-8 once the solve has
converged, and the Krylov value of the same number of steps within 1e-5 (FP32 basis) before that."""
import numpy as np
import pytest

import qudrip_gb300 as q
from qudrip_gb300 import chains

pytestmark = pytest.mark.gpu


def instances(sizes, seed):
    rng = np.random.default_rng(seed)
    hams, v0s = [], []
    for i, (L, n) in enumerate(sizes):
        spec, ham = chains.xxz_chain(L, 1.0, 1.0, True, rng.uniform(-2, 2, L))
        sec = q.Sector(spec.index, [q.getNset(spec.index) == n])
        H = sec.lower(ham)
        H._keep = sec
        hams.append(H)
        v0s.append(q.start_vector(sec.dim, 900 + i))
    return hams, v0s


def krylov_value(H, v0, steps):
    """Lowest eigenvalue of H on the Krylov space of v0 with `steps` vectors (fewer when it is exhausted)."""
    M = H.scipy().real.tocsr()
    V = [v0 / np.linalg.norm(v0)]
    al, be = [], []
    for _ in range(steps):
        w = M @ V[-1]
        al.append(V[-1] @ w)
        for _ in range(2):
            for v in V:
                w = w - (v @ w) * v
        nr = np.linalg.norm(w)
        if nr < 1e-10 or len(V) == H.dim:
            break
        be.append(nr)
        V.append(w / nr)
    k = len(al)
    return np.linalg.eigvalsh(np.diag(al) + np.diag(be[:k - 1], 1) + np.diag(be[:k - 1], -1))[0]


@pytest.mark.parametrize("count,dim,atmost", [
    (30, (16, 8), 8),          # 12,870 rows
    (49, (16, 8), 8),
    (70, (16, 7), 4),          # 11,440
    (98, (16, 8), 3),
    (145, (16, 7), 2),
    (160, (16, 8), 1),
    (20, (17, 8), 8),          # 24,310
])
def test_every_cluster_size(ctx, count, dim, atmost):
    hams, v0s = instances([dim] * count + [(8, 4)], count)
    out = q.batch_lanczos(hams, v0s, 70)
    # as many CTAs as the slots give each (fewer where whole clusters do not fit the GPCs), one for small dimensions
    widths = set(int(w) for w in out[:-1, 7])
    assert len(widths) == 1 and atmost // 2 <= min(widths) and max(widths) <= atmost and out[-1, 7] == 1
    for i in (0, count // 2, count - 1, count):
        e = krylov_value(hams[i], v0s[i], 70)
        assert abs(out[i, 1] - e) <= 1e-8 * abs(e), (i, out[i], e)


@pytest.mark.parametrize("steps", [1, 2, 3, 17, 256])
def test_step_counts_and_exhausted_spaces(ctx, steps):
    hams, v0s = instances([(3, 0), (4, 1), (6, 3), (9, 4), (13, 6), (16, 8)], steps)
    out = q.batch_lanczos(hams, v0s, steps)
    for i, H in enumerate(hams):
        e = krylov_value(H, v0s[i], steps)
        assert abs(out[i, 0] - e) <= 1e-5 * max(1.0, abs(e))
        if steps >= 100:
            assert abs(out[i, 1] - e) <= 1e-8 * max(1.0, abs(e))
