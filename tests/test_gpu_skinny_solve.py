"""The direct solve's kernels (skinny.cu) at their edges.

Leaves of one row up to the largest, odd starts of nodes and panels, 1 to 33
right-hand sides (one tile of 8, two, and the grouped-GEMM form beyond 16),
capacitance systems of less than one 64-row block, of several, and dealt out
over a cluster; in both factorization forms, and through the row-major and the
column-major capacitance solve.  Against the CPU oracle's solution of the same
compressed system, at the tolerance of the repository's other parity tests
(1e-10: two FP64 factorizations of these well-conditioned systems).
"""
import numpy as np
import pytest

from dense_hodlr_b200 import HODLR_Matrix, KernelSpec
from dense_hodlr_b200.points import uniform_1d_sorted, uniform_cube, unit_sphere

from .test_gpu_parity import SOLVE_TOL

pytestmark = pytest.mark.gpu

TYPES = {"gaussian": 0, "matern32": 1}


def _pair(orc, pts, kind, l, shift, leaf, tol):
    n = pts.shape[1]
    g = HODLR_Matrix(n, n, KernelSpec(kind, l, shift), pts, leaf)
    g.set_LRTolerance(tol)
    o = orc.OracleHODLR.from_kernel(pts, TYPES[kind], l, shift=shift, leaf=leaf)
    o.set_lr(tol)
    return g, o


@pytest.mark.parametrize("n,dim,leaf,nrhs", [
    (3, 1, 1, 1), (20, 1, 30, 2), (64, 1, 63, 3), (129, 1, 64, 8), (161, 1, 160, 9),
    (300, 1, 138, 16), (1001, 2, 100, 7), (2047, 2, 65, 17), (5003, 2, 128, 1),
    (5003, 2, 128, 8), (5003, 2, 128, 16), (4096, 2, 64, 33)])
def test_shapes_and_right_hand_sides(oracle_mod, n, dim, leaf, nrhs):
    pts = uniform_1d_sorted(n, -1.0, 1.0, 9) if dim == 1 else uniform_cube(n, dim, 9)
    g, o = _pair(oracle_mod, pts, "matern32" if dim == 2 else "gaussian", 0.2, 0.5, leaf, 1e-8)
    b = np.random.default_rng(nrhs).standard_normal((n, nrhs))
    xo = o.solve(b, nthreads=8)
    for x in (g.recLU_Solve(b), g.recSM_Solve(b)):
        assert np.linalg.norm(x - xo) / np.linalg.norm(xo) <= SOLVE_TOL


@pytest.mark.parametrize("nrhs", [1, 11, 20])
def test_capacitance_over_a_cluster(oracle_mod, nrhs):
    n = 6000
    g, o = _pair(oracle_mod, unit_sphere(n, 12), "matern32", 0.3, 1.0, 128, 1e-8)
    b = np.random.default_rng(nrhs).standard_normal((n, nrhs))
    x, xo = g.recLU_Solve(b), o.solve(b, nthreads=8)
    r = g.ranks()
    assert r[0] + r[1] >= 4 * 64  # several block rows: dealt out over CTAs
    assert np.linalg.norm(x - xo) / np.linalg.norm(xo) <= SOLVE_TOL


def test_counts_change_between_solves_and_logdet(oracle_mod):
    n = 3001
    g, o = _pair(oracle_mod, uniform_cube(n, 2, 13), "matern32", 0.2, 0.5, 128, 1e-9)
    rng = np.random.default_rng(1)
    for nrhs in (8, 1, 16, 40, 2, 40, 1):
        b = rng.standard_normal((n, nrhs))
        xo = o.solve(b, nthreads=8)
        x = g.recLU_Solve(b)
        assert np.linalg.norm(x - xo) / np.linalg.norm(xo) <= SOLVE_TOL
    # the stored triangles are inverted: the log-determinant still is K's
    p = uniform_cube(n, 2, 13)
    d = np.sqrt(((p[:, :, None] - p[:, None, :]) ** 2).sum(0)) * np.sqrt(3.0) / 0.2
    sign, ld = np.linalg.slogdet((1.0 + d) * np.exp(-d) + 0.5 * np.eye(n))
    gs, gl = g.slogdet()
    assert gs == sign and abs(gl - ld) <= 1e-6 * abs(ld)
