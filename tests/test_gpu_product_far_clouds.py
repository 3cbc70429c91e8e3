"""Entries of the row-by-row and forest products for clouds far from the origin.

Points are offset by 1e6 to 1e9 length scales, as timestamps or map coordinates
are; coordinates are multiples of 2^-20, so they and their differences are exact
and the entries are those of the cloud at the origin.  Products with unit vectors
return columns of K; against extended precision with a bound that holds the
cloud's extent (4 length scales a dimension) and not its place.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
N, NRHS = 700, 3


def _cloud(dim, offset):
    rng = np.random.default_rng(dim)
    P = rng.integers(0, 4 << 20, (dim, N)) / 2.0 ** 20
    P[:, N - 2] = P[:, 3]
    return P, P + offset


def _reference(kind, P, cols, shift):
    P = P.astype(np.longdouble)
    d = P[:, :, None] - P[:, None, cols]
    r2 = (d * d).sum(0)
    if kind == "matern32":
        x = np.sqrt(3 * r2)
        K = (1 + x) * np.exp(-x)
    else:
        x = np.sqrt(r2) if kind == "exponential" else r2
        K = (np.exp(-x) if kind in ("gaussian", "exponential")
             else 1 / np.sqrt(1 + x) if kind == "inv_multiquadric" else 1 + x)
    for q, j in enumerate(cols):
        K[j, q] = 1 + np.longdouble(shift)
    # a distance's error: 8 u of the extent (4, and 3^1/2 of it), twice that and the
    # distance itself in a square; 12 u of x and 8 u of the entry on top
    x, K = x.astype(float), K.astype(float)
    e = 8 * U * 4 * 3 ** 0.5 * P.shape[0] ** 0.5
    dx = (e if kind in ("matern32", "exponential") else 2 * np.sqrt(x) * e + e * e) + 12 * U * x
    rel = (dx / (1 + x) if kind in ("inv_multiquadric", "quadratic") else dx) + 8 * U
    return K, rel * np.abs(K) + 1e-300


@pytest.mark.parametrize("form", ["forest", "caller's buffers"])
@pytest.mark.parametrize("offset", [0.0, 2.0 ** 20, 2.0 ** 30])
@pytest.mark.parametrize("dim", [1, 3])
@pytest.mark.parametrize("kind", ["gaussian", "matern32", "exponential", "inv_multiquadric",
                                  "quadratic"])
def test_entries_do_not_depend_on_the_place(kind, dim, offset, form):
    import torch
    from dense_hodlr_b200 import HODLR_Matrix, KernelSpec, _lib

    P, far = _cloud(dim, offset)
    cols = [3, 256, N - 1]
    E = np.zeros((NRHS, N))
    for q, j in enumerate(cols):
        E[q, j] = 1.0
    b = torch.from_numpy(E).cuda()
    y = torch.empty_like(b)
    spec = KernelSpec(kind, 1.0, 0.25)
    torch.cuda.synchronize()
    if form == "caller's buffers":
        p = torch.from_numpy(np.ascontiguousarray(far)).cuda()
        torch.cuda.synchronize()
        assert _lib.lib().hodlr_kernel_matvec_noalloc(
            N, dim, ctypes.c_void_p(p.data_ptr()), ctypes.byref(spec.desc()), NRHS,
            ctypes.c_void_p(b.data_ptr()), N, ctypes.c_void_p(y.data_ptr()), N, None) == 0
    else:
        h = HODLR_Matrix.forest([(far, spec)], leaf=64)
        h.kernel_matvec_device(b.data_ptr(), y.data_ptr(), NRHS)
    torch.cuda.synchronize()
    K, bound = _reference(kind, P, cols, 0.25)
    err = np.abs(y.cpu().numpy().T - K)
    assert np.all(err <= bound), float((err / bound).max())
