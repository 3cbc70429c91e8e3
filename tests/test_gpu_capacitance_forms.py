"""The capacitance solve's forms: a CTA with two column tiles, a CTA per tile, a
cluster, and rows in device memory, which systems of more than 22528 rows take (a
limit on the shared memory makes small ones take it).  All do the same operations
in the same order, so the solutions have the same bits.
"""
import numpy as np
import pytest

from dense_hodlr_b200 import HODLR_Matrix, KernelSpec
from dense_hodlr_b200.points import unit_sphere

pytestmark = pytest.mark.gpu

N = 5001
PTS = unit_sphere(N, 3)


def _handle(limit, monkeypatch):
    if limit:
        monkeypatch.setenv("HODLR_CAPACITANCE_SMEM", str(limit))
    else:
        monkeypatch.delenv("HODLR_CAPACITANCE_SMEM", raising=False)
    g = HODLR_Matrix(N, N, KernelSpec("matern32", 0.2, 0.5), PTS, 100)
    g.set_LRTolerance(1e-8)
    return g


@pytest.mark.parametrize("limit", [1, 60000, 80000])
def test_forms_agree(monkeypatch, limit):
    g, small = _handle(0, monkeypatch), _handle(limit, monkeypatch)
    rng = np.random.default_rng(1)
    for nrhs in (1, 8, 9, 16, 20, 33):
        b = np.asfortranarray(rng.standard_normal((N, nrhs)))
        for f in ("recLU_Solve", "recSM_Solve") if nrhs in (8, 16) else ("recLU_Solve",):
            assert np.array_equal(getattr(small, f)(b), getattr(g, f)(b)), (nrhs, f)
    r = g.ranks()
    assert r[0] + r[1] > 8 * 64  # several block rows a CTA of a cluster of 8
