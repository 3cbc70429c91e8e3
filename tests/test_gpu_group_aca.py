"""The group ACA (aca_group_kernel) against per-thread panel loads (aca_kernel).

The same pivots, ranks and iteration counts on every block and the same W/V
bits on the upper ones, at the sizes where the launch can go wrong: slices of a
few rows, of one chunk and of several, one CTA a block and groups, an odd N
(padded columns), stored matrices, uneven systems in one launch, rank bounds,
skipped rows, and capacities that make blocks pause and resume in the middle.
"""
import numpy as np
import pytest

from dense_hodlr_b200 import HODLR_Matrix, KernelSpec
from dense_hodlr_b200.points import uniform_1d_sorted, uniform_cube, unit_sphere

pytestmark = pytest.mark.gpu


def _same(make, caps=None, factors=6):
    out = []
    for mode in (0, 2):
        g = make()
        g.set_aca_streaming(mode)
        if caps is not None and mode == 2:
            g.set_capacity_hint([caps] * 40)
        g.storeLRinTree()
        nb = g.num_blocks()
        out.append((g.ranks(), [g.block_info(b)["iters"] for b in range(nb)],
                    [g.pivots(b) for b in range(nb)],
                    [g.lowrank(b) for b in range(min(nb, factors))]))
    (r0, i0, p0, f0), (r1, i1, p1, f1) = out
    assert np.array_equal(r0, r1)
    assert i0 == i1
    for a, b in zip(p0, p1):
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    for (W0, V0), (W1, V1) in zip(f0, f1):
        assert np.array_equal(W0, W1) and np.array_equal(V0, V1)


@pytest.mark.parametrize("n,dim,kind,l,leaf,tol", [
    (65, 1, "gaussian", 0.1, 32, 1e-10), (131, 2, "matern32", 0.3, 64, 1e-8),
    (1023, 2, "exponential", 0.2, 30, 1e-6), (4097, 1, "gaussian", 0.1, 64, 1e-10),
    (20011, 2, "matern32", 0.2, 128, 1e-8), (9001, 3, "inv_multiquadric", 0.5, 100, 1e-8),
    (150001, 1, "matern32", 0.05, 128, 1e-10)])
def test_kernel_systems(n, dim, kind, l, leaf, tol):
    pts = uniform_1d_sorted(n, -1.0, 1.0, 3) if dim == 1 else uniform_cube(n, dim, 3)

    def make():
        g = HODLR_Matrix(n, n, KernelSpec(kind, l, 0.1), pts, leaf)
        g.set_LRTolerance(tol)
        return g
    _same(make)


@pytest.mark.parametrize("n,caps", [(6001, 1), (6001, 17), (40000, 40)])
def test_blocks_pause_and_resume(n, caps):
    pts = uniform_cube(n, 2, 4) if n < 40000 else unit_sphere(n, 4)

    def make():
        g = HODLR_Matrix(n, n, KernelSpec("matern32", 0.3, 0.1), pts, 128)
        g.set_LRTolerance(1e-6)
        return g
    _same(make, caps=caps)


def test_uneven_systems_share_launches():
    rng = np.random.default_rng(5)
    systems = [(uniform_1d_sorted(int(n), 0.0, 1.0, int(n)), KernelSpec("gaussian", 0.2, 1.0))
               if q % 2 else (uniform_cube(int(n), 2, int(n)), KernelSpec("matern32", 0.3, 0.5))
               for q, n in enumerate(rng.integers(150, 9000, 9))]

    def make():
        g = HODLR_Matrix.forest(systems, leaf=50)
        g.set_LRTolerance(1e-8)
        return g
    _same(make)


@pytest.mark.parametrize("min_pivot", [0.0, 2.5])
def test_stored_matrix_and_skipped_rows(min_pivot):
    x = uniform_1d_sorted(1777, -1.0, 1.0, 8)[0]
    A = 10.0 * np.exp(-((x[:, None] - x[None, :]) / 0.1) ** 2) + np.eye(len(x))

    def make():
        g = HODLR_Matrix(A, 48)
        g.set_LRTolerance(1e-10)
        g.set_minPivot(min_pivot)
        return g
    _same(make)


@pytest.mark.parametrize("bounds", [(3, 3, 5, 5), (40, 40, -1, -1), (-1, -1, 1, 1), (-1, -1, 2, 0)])
def test_rank_bounds(bounds):
    n = 4000
    pts = uniform_cube(n, 2, 6)

    def make():
        g = HODLR_Matrix(n, n, KernelSpec("matern32", 0.2, 0.1), pts, 64)
        g.set_LRTolerance(1e-8)
        g.set_index_tree([n // 2], [-1], [-1], [[b] for b in bounds])
        return g
    _same(make)
