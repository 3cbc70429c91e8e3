"""A compression is the same to the last bit every time.

Blocks that pause in the middle go on in groups of another size, so when they pause
must not depend on the clock: ranks, iteration counts and the distance of every
epsilon from the tolerance are compared over repeated compressions, of systems
large enough to pause.
"""
import numpy as np
import pytest

from dense_hodlr_b200 import HODLR_Matrix, KernelSpec
from dense_hodlr_b200.points import uniform_cube, unit_sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cloud,n,kind,l,tol", [
    ("sphere", 16384, "matern32", 0.1, 1e-10), ("square", 30001, "matern32", 0.2, 1e-9)])
def test_same_bits_every_time(cloud, n, kind, l, tol):
    pts = unit_sphere(n, 1) if cloud == "sphere" else uniform_cube(n, 2, 1)
    seen = []
    for _ in range(4):
        g = HODLR_Matrix(n, n, KernelSpec(kind, l, 0.1), pts, 128)
        g.set_LRTolerance(tol)
        g.storeLRinTree()
        nb = g.num_blocks()
        seen.append((list(g.ranks()), [g.block_info(b)["iters"] for b in range(nb)],
                     [g.margin(b) for b in range(nb)], g.aca_stats()["launches"]))
    assert all(s == seen[0] for s in seen)
