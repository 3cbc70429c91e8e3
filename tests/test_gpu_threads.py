"""Handles of different sizes in threads at the same time.

Kernels whose shared memory depends on the problem (ACA rings, LU panels, the
solves' rows) are launched by all of them with sizes of their own; ctypes releases
the interpreter lock during calls.  Each result is that of the handle alone.
"""
import threading

import numpy as np
import pytest

from dense_hodlr_b200 import HODLR_Matrix, KernelSpec
from dense_hodlr_b200.points import uniform_cube

pytestmark = pytest.mark.gpu

# (points, leaf, tolerance, right-hand sides)
SIZES = [(300, 30, 1e-4, 1), (700, 64, 1e-6, 9), (1500, 100, 1e-8, 1), (2500, 128, 1e-9, 16),
         (600, 40, 1e-10, 20), (3500, 128, 1e-10, 3), (900, 138, 1e-5, 8), (2000, 50, 1e-7, 12)]


def _solve(q):
    n, leaf, tol, nrhs = SIZES[q]
    g = HODLR_Matrix(n, n, KernelSpec("matern32", 0.3, 0.5), uniform_cube(n, 2, q), leaf)
    g.set_LRTolerance(tol)
    return np.array(g.recLU_Solve(np.random.default_rng(q).standard_normal((n, nrhs))))


def test_threads_with_different_shared_memory():
    want = [_solve(q) for q in range(len(SIZES))]
    failures = []
    start = threading.Barrier(len(SIZES))

    def work(q):
        try:
            start.wait()
            for r in range(12):
                k = (q + r) % len(SIZES)
                x = _solve(k)
                if not np.allclose(x, want[k], rtol=0, atol=1e-10 * np.abs(want[k]).max()):
                    failures.append((k, np.abs(x - want[k]).max()))
        except Exception as e:
            failures.append((q, repr(e)))

    threads = [threading.Thread(target=work, args=(q,)) for q in range(len(SIZES))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
