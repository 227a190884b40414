"""Two threads, each with its own context, run the persistent Krylov kernels at different sizes: the limit of
a kernel's dynamic shared memory is shared by all launches of the process."""
import threading

import numpy as np
import pytest

import qudrip_gb300 as q
from qudrip_gb300 import chains

pytestmark = pytest.mark.gpu


def test_sizes_of_other_threads_do_not_limit_a_launch():
    errors = []

    def work(L):
        c = q.Context(0)
        try:
            spec, ham = chains.xxz_chain(L, 1.0, 0.7, True, np.linspace(-1, 1, L))
            sec = q.Sector(spec.index, spec.constraints, spec.tight, ctx=c)
            H = sec.lower(ham)
            rng = np.random.default_rng(L)
            x = rng.normal(size=sec.dim) + 1j * rng.normal(size=sec.dim)
            psi = q.getState(sec, 2)
            solver = q.Arnoldi.getSolver(sec, 20)
            want = {}
            for _ in range(40):
                psi.set(0, x)
                psi.set(1, x)
                solver.evolve_inplace(H, psi, 0, 0.05)
                q.lanczos_evolve(H, psi, 1, 1, 0.05, 20)
                for t in (0, 1):
                    got = psi.get(t)
                    assert np.array_equal(got, want.setdefault(t, got))
            assert np.linalg.norm(want[0] - want[1]) < 1e-12
            del psi, solver, H, sec
        except BaseException as e:  # noqa: BLE001
            errors.append((L, e))
        finally:
            c.close()

    ts = [threading.Thread(target=work, args=(L,)) for L in (9, 12, 15)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errors, errors
