"""Backward stability of the direct solve (skinny.cu) on ill-conditioned systems.

The triangles of the stored LUs are applied as inverses, refined by their
condition; the residual on the compressed operator is compared with that of the
CPU oracle, which substitutes, both over the norms of their solutions (backward
errors: at a shift of 1e-12 the solutions have few digits in common).  Unrefined
inverses left 1.3 to 112 times the oracle's.  By the rule of the kernels a block
step leaves at most 1.4 times a substitution's residual; 3 allows for the scatter
of residuals of 24 random columns.
"""
import numpy as np
import pytest

from dense_hodlr_b200 import HODLR_Matrix, KernelSpec
from dense_hodlr_b200.points import uniform_1d_sorted, uniform_cube

pytestmark = pytest.mark.gpu

TYPES = {"gaussian": 0, "matern32": 1}


def _apply(g, o, x):
    """K_H x: W V^T on the off-diagonal blocks, on the leaves the kernel's entries
    as both sides have them (the oracle's: another exponential's rounding would
    show in the residual of a condition above 1e12)."""
    y = np.zeros_like(x)
    edges = {0, g.n}
    for q in range(g.num_blocks()):
        i = g.block_info(q)
        W, V = g.lowrank(q)
        y[i["row0"]:i["row0"] + i["m"]] += W @ (V.T @ x[i["col0"]:i["col0"] + i["n"]])
        edges |= {i["row0"], i["col0"]}
    edges = sorted(edges)
    for s, e in zip(edges[:-1], edges[1:]):
        K = np.array([[o.entry(i, j) for j in range(s, e)] for i in range(s, e)])
        y[s:e] += K @ x[s:e]
    return y


SYSTEMS = [("leaf", 128, 1, "gaussian", 0.1, 140), ("1d", 1024, 1, "gaussian", 0.1, 64),
           ("2d", 2001, 2, "matern32", 0.2, 100)]


@pytest.mark.parametrize("nrhs", [1, 8, 20])
@pytest.mark.parametrize("name,n,dim,kind,l,leaf,shift", [
    s + (shift,) for s in SYSTEMS for shift in (1e-2, 1e-4, 1e-6, 1e-8, 1e-10, 1e-12)
    if shift >= 1e-8 or s[0] == "leaf"])  # below: the accuracy of the compression
def test_residual_is_a_substitutions(oracle_mod, name, n, dim, kind, l, leaf, shift, nrhs):
    pts = uniform_1d_sorted(n, -1.0, 1.0, 3) if dim == 1 else uniform_cube(n, dim, 3)
    g = HODLR_Matrix(n, n, KernelSpec(kind, l, shift), pts, leaf)
    g.set_LRTolerance(1e-10)
    o = oracle_mod.OracleHODLR.from_kernel(pts, TYPES[kind], l, shift=shift, leaf=leaf)
    o.set_lr(1e-10)
    b = np.asfortranarray(np.random.default_rng(4).standard_normal((n, 24)))
    x = np.hstack([np.asarray(g.recLU_Solve(np.asfortranarray(b[:, c:c + nrhs]))).reshape(n, -1)
                   for c in range(0, 24, nrhs)])
    xo = o.solve(b, nthreads=8)
    r = np.linalg.norm(b - _apply(g, o, x)) / np.linalg.norm(x)
    ro = np.linalg.norm(b - _apply(g, o, xo)) / np.linalg.norm(xo)
    print(f"{name} shift {shift:g} nrhs {nrhs}: {r / ro:.2f} of the oracle's {ro:.1e}")
    assert r <= 3.0 * ro


@pytest.mark.parametrize("e", [-1015, -500, 500, 1005])
def test_scaled_by_a_power_of_two(e):
    """Pivots whose reciprocals leave the range of normal numbers."""
    rng = np.random.default_rng(8)
    A = 0.1 * rng.standard_normal((128, 128)) + 2.0 * np.eye(128)
    x = rng.standard_normal((128, 3))
    b = A @ x
    for s in (1.0, 2.0 ** e):
        h = HODLR_Matrix(np.asfortranarray(A * s), 140)
        got = np.asarray(h.recLU_Solve(np.asfortranarray(b * s)))
        # condition below 10, 128 u: 1e-12 leaves a factor of 10
        assert np.abs(got - x).max() <= 1e-12
        sign, ld = h.slogdet()
        want = np.linalg.slogdet(A)
        assert sign == want[0] and abs(ld - want[1] - 128 * np.log(s)) <= 1e-9
