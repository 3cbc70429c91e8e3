"""A group launch whose faster form has no room for a ring beside its columns.

With capacities of 8400 columns the coefficients and dots of the 8 x 1 form leave
less than three stages; the 8 x 4 form streams such blocks (before, they fell back
to panels loaded per thread).  The same pivots, ranks and factors as that form.
"""
import numpy as np
import pytest

from dense_hodlr_b200 import HODLR_Matrix, KernelSpec
from dense_hodlr_b200.points import uniform_cube

pytestmark = pytest.mark.gpu


def test_more_columns_than_fit_beside_the_ring():
    n = 17001
    pts = uniform_cube(n, 2, 2)
    out = []
    for mode in (0, 2):
        g = HODLR_Matrix(n, n, KernelSpec("matern32", 0.2, 0.1), pts, 128)
        g.set_LRTolerance(1e-6)
        g.set_aca_streaming(mode)
        g.set_capacity_hint([8400])
        g.storeLRinTree()
        nb = g.num_blocks()
        out.append((g.ranks(), [g.pivots(b) for b in range(nb)], g.lowrank(0), g.lowrank(1)))
    (r0, p0, a0, b0), (r1, p1, a1, b1) = out
    assert np.array_equal(r0, r1)
    for p, q in zip(p0, p1):
        assert np.array_equal(p[0], q[0]) and np.array_equal(p[1], q[1])
    for (W, V), (X, Y) in ((a0, a1), (b0, b1)):
        assert np.array_equal(W, X) and np.array_equal(V, Y)
