"""Row-major dense input is transposed on the device; pinned staging blocks
pass from handle to handle.  Both only move bytes, so results are compared
bit for bit with the column-major and the one-at-a-time runs."""
import threading

import numpy as np
import pytest

from dense_hodlr_b200 import HODLR_Matrix, KernelSpec

pytestmark = pytest.mark.gpu


def _solve(A, b, leaf=30):
    h = HODLR_Matrix(A, leaf)
    h.set_LRTolerance(1e-8)
    return h.recLU_Solve(b)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 257])
def test_row_major_is_column_major(n):
    rng = np.random.default_rng(n)
    x = np.sort(rng.uniform(-1, 1, n))
    A = np.exp(-np.abs(x[:, None] - x[None, :] * 0.9)) + np.diag(rng.uniform(1, 2, n))  # unsymmetric
    b = rng.standard_normal(n)
    C, F = np.ascontiguousarray(A), np.asfortranarray(A)
    got, want = _solve(C, b), _solve(F, b)
    assert np.array_equal(got, want)
    assert np.array_equal(C, A)


def test_handles_in_threads_share_staging():
    cases = []
    for q in range(6):
        rng = np.random.default_rng(q)
        n = 700 + 211 * q
        cases.append((np.sort(rng.uniform(-1, 1, n))[None], rng.standard_normal(n)))

    def solve(q):
        pts, b = cases[q]
        h = HODLR_Matrix(pts.shape[1], pts.shape[1], KernelSpec("gaussian", 0.1, diag_shift=1.0), pts, 64)
        h.set_LRTolerance(1e-10)
        return h.recLU_Solve(b)

    want = [solve(q) for q in range(6)]
    got = [[] for _ in range(6)]

    def work(q):
        for _ in range(3):
            got[q].append(solve(q))

    threads = [threading.Thread(target=work, args=(q,)) for q in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for q in range(6):
        assert len(got[q]) == 3
        for x in got[q]:
            assert np.array_equal(x, want[q])
