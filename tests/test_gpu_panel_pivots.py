"""Capacitance LUs whose accuracy hangs on the pivots.

Dense matrices with unit leaves and full-rank off-diagonal blocks of entries near
1e6: the capacitance matrices are [[I, A], [B, I]] with A and B of that size.
Eliminating with the ones on the diagonal grows entries to 1e12 and more and loses
as many digits of the identity (numpy, 258 rows: backward error 2.7e-7 against
1.6e-16 with pivoting).  Against the oracle, which runs the same algorithm with
partial pivoting.  Sizes cross the panels' forms: one CTA (32 columns), one CTA
and clusters a panel (512 rows each), pivots in every CTA of a cluster.
"""
import numpy as np
import pytest

from dense_hodlr_b200 import HODLR_Matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaf", [(40, 30), (66, 64), (250, 128), (258, 130), (514, 130),
                                    (1040, 130), (1100, 138), (2100, 132)])
@pytest.mark.parametrize("ties", [False, True])
def test_pivots_keep_the_digits(oracle_mod, n, leaf, ties):
    rng = np.random.default_rng(n)
    A = rng.choice([-1.0, 1.0], (n, n)) if ties else rng.standard_normal((n, n))
    A *= 1e6
    h = n // 2  # the root's blocks; all others are zero and the leaves unit matrices
    for s in (slice(0, h), slice(h, n)):
        A[s, s] = np.eye(s.stop - s.start)
    x = rng.standard_normal((n, 2))
    b = A @ x
    g = HODLR_Matrix(np.asfortranarray(A), leaf)
    g.set_LRTolerance(1e-15)
    got = np.asarray(g.recLU_Solve(np.asfortranarray(b))).reshape(n, 2)
    o = oracle_mod.OracleHODLR.from_dense(A, leaf=leaf)
    o.set_lr(1e-15)
    ref = o.solve(b, nthreads=8)

    def backward(y):
        return np.linalg.norm(b - A @ y) / (np.linalg.norm(A) * np.linalg.norm(y))

    # growth and summation order differ between the two within a factor of ten
    print(n, ties, backward(got), backward(ref))
    assert backward(got) <= 10.0 * backward(ref) + 1e-16
