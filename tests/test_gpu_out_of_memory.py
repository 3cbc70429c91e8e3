"""Calls that run out of device memory, under a limit that the host keeps.

A call that does not fit returns HODLR_ERR_ALLOC and may be repeated: at the same
limit it fails again or succeeds with the right answer (no kernel runs on a buffer
that is not there), and without the limit it succeeds.  The limits step through
what the call takes, so that each of its allocations is the one that fails.
"""
import numpy as np
import pytest

from dense_hodlr_b200 import HODLR_Matrix, HODLRError, KernelSpec, _lib
from dense_hodlr_b200.points import uniform_cube

pytestmark = pytest.mark.gpu

N = 3001
PTS = uniform_cube(N, 2, 5)


def _handle():
    g = HODLR_Matrix(N, N, KernelSpec("matern32", 0.2, 0.5), PTS, 100)
    g.set_LRTolerance(1e-8)
    return g


def _rhs(nrhs):
    return np.asfortranarray(np.random.default_rng(nrhs).standard_normal((N, nrhs)))


def _close(x, ref):
    # the same compression and factors; plans may differ in their split sums
    return np.abs(np.asarray(x).reshape(ref.shape) - ref).max() <= 1e-10 * np.abs(ref).max()


def _attempt(g, b, ref):
    try:
        x = g.recLU_Solve(b)
    except HODLRError as e:
        assert e.status == _lib.ERR_ALLOC
        return False
    assert _close(x, ref)
    return True


def _solved_without_cache(precision, b1, x1):
    """A factored handle that has solved for one column and holds no cached memory:
    a call that cannot fit has given the cache back."""
    g = _handle()
    g.set_precision(precision)
    x = g.recLU_Solve(b1)
    assert x1 is None or _close(x, x1)
    g.set_memory_limit(1)
    with pytest.raises(HODLRError):
        g.recLU_Solve(_rhs(600))
    return g


@pytest.mark.parametrize("precision", ["fp64", "tf32x3"])
@pytest.mark.parametrize("nrhs", [16, 33])
def test_more_right_hand_sides_than_fit(nrhs, precision):
    b1, b = _rhs(1), _rhs(nrhs)
    g = _solved_without_cache(precision, b1, None)
    low = g.memory_held()
    g.set_memory_limit(0)
    x = np.asarray(g.recLU_Solve(b)).reshape(N, nrhs)
    high = g.memory_held()
    x1 = np.asarray(g.recLU_Solve(b1)).reshape(N, 1)
    assert high > low
    failed = 0
    for limit in np.linspace(low, high, 25).astype(int):
        g = _solved_without_cache(precision, b1, x1)
        g.set_memory_limit(limit)
        for _ in range(2):
            failed += not _attempt(g, b, x)
            _attempt(g, b1, x1)
        g.set_memory_limit(0)
        assert _close(g.recLU_Solve(b), x)
        assert _close(g.recLU_Solve(b1), x1)
    assert failed


def test_whole_calls_that_do_not_fit():
    b = _rhs(2)
    g = _handle()
    empty = g.memory_held()
    x = np.asarray(g.recLU_Solve(b)).reshape(N, 2)
    failed = 0
    for limit in np.linspace(empty, g.memory_held(), 40).astype(int):
        g = _handle()
        g.set_memory_limit(limit)
        for _ in range(2):
            failed += not _attempt(g, b, x)
        g.set_memory_limit(0)
        assert _close(g.recLU_Solve(b), x)
    assert failed


@pytest.mark.parametrize("hint", [0, 8])
def test_streamed_compression_fits_where_per_thread_loads_do(hint):
    """The working layout of the group levels is a second copy of their panels: it
    is given back when a level grows (hint: from 8 columns) or another one starts."""
    n = 12001
    pts = uniform_cube(n, 2, 6)

    def compress(mode, limit):
        g = HODLR_Matrix(n, n, KernelSpec("matern32", 0.2, 0.5), pts, 128)
        g.set_LRTolerance(1e-8)
        g.set_aca_streaming(mode)
        if hint:
            g.set_capacity_hint([hint] * 20)
        g.set_memory_limit(limit)
        g.storeLRinTree()
        return g.ranks(), g.memory_held()

    ranks, most = compress(0, 0)
    too_little, enough = most // 8, most  # what per-thread loads need, by bisection
    while enough - too_little > 1 << 18:
        limit = (too_little + enough) // 2
        try:
            assert np.array_equal(compress(0, limit)[0], ranks)
            enough = limit
        except HODLRError as e:
            assert e.status == _lib.ERR_ALLOC
            too_little = limit
    # exchange slots and published rows of the group form: below 4 MB
    for limit in np.linspace(enough + (4 << 20), 2 * most, 40).astype(int):
        assert np.array_equal(compress(2, limit)[0], ranks)
