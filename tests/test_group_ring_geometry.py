"""Index arithmetic of the group ACA's shared ring (csrc/aca_group.cu), on the CPU.

slice_chunks, slice_pitch, make_slice, ring_issue, aca_group_slice and
aca_group_ring restated, and checked over many slice shapes: the CTAs' slices
and their chunks cover a block's rows once and stay inside the working memory
that the launch asks for; every tile starts on a 16-byte boundary, has a
multiple of 16 bytes and fits its stage; and the rings fit the shared memory.
"""
import numpy as np
import pytest

SMAX, SMIN = 16, 3
# (sum warps, rows a thread) -> tile columns, dynamic shared memory of a launch
VARIANTS = {(8, 1): (16, 212 * 1024), (8, 4): (4, 224 * 1024)}


def chunks_of(per, most):
    return (per + most - 1) // most


def pitch(per, most):
    c = chunks_of(per, most)
    return ((per + c - 1) // c + 15) & ~15


def stage_elems(tc, rows, most):
    return tc * min(most, (rows + 15) & ~15)


def ring(rows, kcap, v):
    tc, budget = VARIANTS[v]
    elems = stage_elems(tc, rows, 32 * v[0] * v[1])
    fixed = 8 * (((kcap + 16) & ~15) + (kcap if v[1] == 1 else 0))
    st = 0 if fixed >= budget else min(SMAX, (budget - fixed) // (8 * elems))
    return (st if st >= SMIN else 0), elems, 8 * elems * st + fixed


@pytest.mark.parametrize("v", list(VARIANTS))
def test_slices_chunks_and_copies(v):
    most, tc = 32 * v[0] * v[1], VARIANTS[v][0]
    rng = np.random.default_rng(most)
    shapes = [(1, 1), (2, 1), (31, 1), (most, 1), (most + 1, 1), (2 * most - 1, 1), (2 * most, 1),
              (135, 1), (1771 * 74, 74), (10010, 74), (17, 16), (5, 7)]
    shapes += [(int(rng.integers(1, 9000)), int(rng.integers(1, 150))) for _ in range(300)]
    for m, G in shapes:
        kcap = int(rng.integers(1, 60))
        per = (m + G - 1) // G
        cr = pitch(per, most)
        stride = chunks_of(per, most) * cr * kcap
        assert cr % 16 == 0 and cr <= most
        # a stage is sized for the launch's longest slice
        longest = per + int(rng.integers(0, 3000))
        assert tc * cr <= stage_elems(tc, longest, most)
        seen = np.zeros(m, dtype=int)
        for g in range(G):
            lo = min(m, g * per)
            hi = min(m, lo + per)
            chunks = (hi - lo + cr - 1) // cr
            assert chunks <= chunks_of(per, most)
            for c in range(chunks):
                j = lo + c * cr + np.arange(cr)
                seen[j[j < hi]] += 1
                k = int(rng.integers(1, kcap + 1))
                for l0 in range(0, k, tc):
                    nc = min(tc, k - l0)
                    start = g * stride + (c * kcap + l0) * cr
                    assert (8 * start) % 16 == 0 and (8 * nc * cr) % 16 == 0
                    assert start + nc * cr <= (g + 1) * stride
            for row in range(lo, hi):  # where another CTA looks a row up
                og = row // per
                assert og == g
                oj = row - og * per
                assert oj // cr < chunks and (oj // cr) * cr + oj % cr == row - lo
        assert np.all(seen == 1)


@pytest.mark.parametrize("v", list(VARIANTS))
def test_rings_fit_their_shared_memory(v):
    tc, budget = VARIANTS[v]
    fitted = 0
    for rows in (1, 2, 7, 64, 111, 128, 129, 256, 300, 1771, 131072):
        for kcap in (1, 15, 16, 64, 371, 1352, 2001, 4117, 8192, 20000):
            st, elems, nbytes = ring(rows, kcap, v)
            if st:
                fitted += 1
                assert SMIN <= st <= SMAX and nbytes <= budget
                assert (8 * elems) % 128 == 0  # every stage starts on a 128-byte boundary
                # coefficients are read in pairs up to the end of a tile, past column k
                assert (kcap + 16) & ~15 >= -(-kcap // tc) * tc
    assert fitted
