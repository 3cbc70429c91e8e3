"""Solve plans rebuilt outside the captured graph (one handle, several counts)."""
import numpy as np
import pytest

from dense_hodlr_b200 import HODLR_Matrix, KernelSpec
from dense_hodlr_b200.points import uniform_cube

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("few,many", [(1, 16), (3, 40)])
def test_graph_of_a_plan_that_was_replaced(few, many):
    """All buffers have their full size after the first solve, so nothing but the
    plans tells the captured graph of `few` columns from the one needed after
    checked solves, which use no graph, have built plans for other counts."""
    n = 3000
    g = HODLR_Matrix(n, n, KernelSpec("matern32", 0.2, 0.5), uniform_cube(n, 2, 7), 100)
    g.set_LRTolerance(1e-8)
    rng = np.random.default_rng(3)
    counts = (many, few, many - 1, few + 1)
    b = {q: np.asfortranarray(rng.standard_normal((n, q))) for q in counts}
    x = {q: np.array(g.recLU_Solve(b[q])) for q in counts}
    for _ in range(3):
        assert np.allclose(g.recLU_Solve(b[few]), x[few], rtol=0, atol=1e-10)  # captured
        g.set_checked(True)
        for q in (many, many - 1, few + 1):  # the replaced plan's memory is used again
            assert np.allclose(g.recLU_Solve(b[q]), x[q], rtol=0, atol=1e-10)
        g.set_checked(False)
        assert np.allclose(g.recLU_Solve(b[few]), x[few], rtol=0, atol=1e-10)
