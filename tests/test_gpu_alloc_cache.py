"""Device buffers that a context keeps for its next operators: a new operator in reused buffers equals the
oracle, on one context and on two used by two threads, whatever the order the objects are dropped in."""
import threading

import numpy as np
import pytest

import oracle as O
import qudrip_gb300 as q
from qudrip_gb300 import chains

pytestmark = pytest.mark.gpu


def build_and_check(ctx, L, seed):
    rng = np.random.default_rng(seed)
    spec, ham = chains.xxz_chain(L, 1.0, 0.7, True, rng.uniform(-1, 1, L))
    H = q.Sector(spec.index, spec.constraints, spec.tight, ctx=ctx).lower(ham)
    M = O.Ham(O.Sector(spec), ham).scipy().tocsr()
    M.sort_indices()
    rp, ci, v = H.csr()
    assert np.array_equal(rp, M.indptr) and np.array_equal(ci, M.indices) and np.array_equal(v, M.data)


def test_operators_of_changing_sizes_in_reused_buffers(ctx):
    for k, L in enumerate((12, 6, 12, 9, 3, 12, 9)):
        build_and_check(ctx, L, k)


def test_two_contexts_on_two_threads():
    errors = []

    def work(seed):
        c = q.Context(0)
        try:
            for k in range(6):
                build_and_check(c, 8 + (k + seed) % 4, 10 * seed + k)
        except BaseException as e:  # noqa: BLE001
            errors.append(e)
        finally:
            c.close()

    ts = [threading.Thread(target=work, args=(s,)) for s in (1, 2)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errors, errors


def test_objects_dropped_in_any_order_and_on_another_thread():
    c = q.Context(0)
    spec, ham = chains.xxz_chain(10, 1.0, 0.7, True)
    S = q.Sector(spec.index, spec.constraints, spec.tight, ctx=c)
    held = [S.lower(ham) for _ in range(3)]
    t = threading.Thread(target=held.clear)
    t.start()
    t.join()
    build_and_check(c, 10, 3)
