"""LU panels of a cluster of CTAs, many clusters in one launch.

Systems on a sphere whose top capacitance matrices have more than 512 rows, so
that their panels run on clusters that write each other's shared memory, two
dozen at a time.  Against dense solves: blocks are compressed to 1e-10 and the
condition is below 1e3 (kernel sums below 1e3, shift 1), so 1e-6 leaves a factor
of ten; a lost candidate or pivot row is off by O(1).
"""
import numpy as np
import pytest

from dense_hodlr_b200 import HODLR_Matrix, KernelSpec
from dense_hodlr_b200.points import unit_sphere

pytestmark = pytest.mark.gpu


def test_many_clusters_at_once():
    sizes = [2400 + 67 * q for q in range(24)]
    pts = [unit_sphere(n, n) for n in sizes]
    g = HODLR_Matrix.forest([(p, KernelSpec("matern32", 0.1, 1.0)) for p in pts], leaf=128)
    g.set_LRTolerance(1e-10)
    b = np.random.default_rng(2).standard_normal((sum(sizes), 1))
    x = np.asarray(g.recLU_Solve(b)).reshape(-1)
    info = [g.block_info(q) for q in range(g.num_blocks())]
    # the roots' capacitance matrices have the ranks of both off-diagonal blocks
    top = [i["rank"] for i in info if i["level"] == 0]
    assert len(top) == 2 * len(sizes) and min(top) > 256
    o = 0
    for p, n in zip(pts, sizes):
        d = np.sqrt(np.maximum(((p[:, :, None] - p[:, None, :]) ** 2).sum(0), 0.0)) * np.sqrt(3.0) / 0.1
        K = (1.0 + d) * np.exp(-d) + np.eye(n)
        assert np.abs(K).sum(1).max() < 1e3
        ref = np.linalg.solve(K, b[o:o + n, 0])
        assert np.abs(x[o:o + n] - ref).max() <= 1e-6 * np.abs(ref).max()
        o += n
