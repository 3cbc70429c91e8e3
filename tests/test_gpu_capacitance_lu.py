"""Partial-pivot LU of the capacitance matrices at the edges of its forms: one
32-column panel and its neighbours, the one-CTA and multi-CTA kernels around
their threshold, one CTA or a cluster of them for a panel (512 rows each), and
the shared-memory panels above 4096 rows.

A dense matrix with random off-diagonal blocks has full-rank blocks, so the top
node's capacitance matrix has n rows.  With a diagonal of 4 and off-diagonal
entries N(0, 1/n) the condition number is below 10; cross approximation of a
random block may grow errors by some thousands, n u is below 1e-12: 1e-8 covers
both with a factor to spare, and a wrong pivot, move or update is off by O(1).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(n, seed, ties):
    rng = np.random.default_rng(seed)
    if ties:  # entries of equal magnitude: every pivot search is a tie
        A = rng.choice([-1.0, 1.0], (n, n)) / np.sqrt(n)
    else:
        A = rng.standard_normal((n, n)) / np.sqrt(n)
    return A + 4.0 * np.eye(n)


@pytest.mark.parametrize("n,leaf,ties", [
    (31, 20, False), (32, 20, False), (33, 20, False), (64, 40, True), (65, 40, False),
    (130, 70, True), (255, 80, False), (256, 80, False), (257, 80, True), (385, 100, True), (512, 128, False),
    (513, 130, False), (545, 130, True), (1056, 130, False), (1537, 128, False),
    (2600, 128, False), (4230, 133, False)])
def test_capacitance_lu(n, leaf, ties):
    from dense_hodlr_b200 import HODLR_Matrix

    A = _matrix(n, n, ties)
    rng = np.random.default_rng(1)
    x = rng.standard_normal((n, 2))
    h = HODLR_Matrix(np.asfortranarray(A), leaf)
    h.set_LRTolerance(1e-15)
    got = np.asarray(h.recLU_Solve(np.asfortranarray(A @ x))).reshape(n, 2)
    assert np.abs(got - x).max() <= 1e-8 * np.abs(x).max()
