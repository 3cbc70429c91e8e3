"""Entries of the full-kernel product against extended precision.

The product with unit vectors returns columns of K exactly (all other terms are
zeros), so each entry can be compared by itself.  Sizes cross the 256-point
tiles; length scales reach from nearly constant kernels to entries that
underflow; two points coincide.
"""
import os
import re

import numpy as np
import pytest

U = 2.0 ** -53


def test_exponential_table_correctly_rounded():
    from decimal import Decimal, getcontext
    getcontext().prec = 60
    path = os.path.join(os.path.dirname(__file__), "..", "dense_hodlr_b200", "csrc", "exp2_table.inc")
    got = [float.fromhex(x) for x in re.findall(r"0x1\.[0-9a-f]{13}p[+-]\d", open(path).read())]
    assert len(got) == 2048
    for j in range(0, 2048):
        assert got[j] == float(Decimal(2) ** (Decimal(-j) / 2048)), j


def _reference(kind, dim, l, P, cols, shift):
    P = P.astype(np.longdouble)
    d = P[:, :, None] - P[:, None, cols]
    r2 = (d * d).sum(0)
    l = np.longdouble(l)
    if kind == "gaussian":
        x = r2 / (l * l)
        K = np.exp(-x)
    elif kind in ("matern32", "exponential"):
        x = np.sqrt(r2) / l
        if kind == "matern32":
            x = x * np.sqrt(np.longdouble(3))
        K = (1 + x) * np.exp(-x) if kind == "matern32" else np.exp(-x)
    else:
        x = r2 / (l * l)
        K = 1 / np.sqrt(1 + x) if kind == "inv_multiquadric" else 1 + x
    for q, j in enumerate(cols):
        K[j, q] = 1 + np.longdouble(shift)
    return K, x


def _bound(kind, dim, l, P, K, x):
    # x is formed from coordinates scaled in double: each carries up to 4 u of
    # its largest scaled value C, the differences and the sum of squares 8 u more
    C = float(np.abs(P).max()) / l * (3 ** 0.5 if kind == "matern32" else 1.0)
    x = x.astype(float)
    K = K.astype(float)
    e = 8 * U * dim ** 0.5 * C  # in the distance
    if kind in ("matern32", "exponential"):
        dx = e + 8 * U * x
        rel = dx + 8 * U
    elif kind == "gaussian":
        dx = 2 * np.sqrt(x) * e + e * e + 12 * U * x
        rel = dx + 8 * U
    else:
        dx = 2 * np.sqrt(x) * e + e * e + 12 * U * x
        rel = dx / (1 + x) + 8 * U
    return rel * K + 1e-300


@pytest.mark.gpu
@pytest.mark.parametrize("nrhs", [1, 3, 8, 11])
@pytest.mark.parametrize("n", [255, 257, 700, 10753])  # 10753: 903 tile pairs, 4 rows a thread
@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("kind", ["gaussian", "matern32", "inv_multiquadric", "quadratic",
                                  "exponential"])
def test_entries(kind, dim, n, nrhs):
    import torch
    from dense_hodlr_b200 import HODLR_Matrix, KernelSpec

    rng = np.random.default_rng(dim * 1000 + n + nrhs)
    P = rng.uniform(0, 1, (dim, n))
    P[:, n - 2] = P[:, 3]
    cols = [int(c) for c in rng.choice(n, nrhs, replace=False)]
    cols[0] = 3
    if len(set(cols)) < nrhs:
        cols = list(range(3, 3 + nrhs))
    E = np.zeros((nrhs, n))
    for q, j in enumerate(cols):
        E[q, j] = 1.0
    b = torch.from_numpy(E).cuda()
    y = torch.empty_like(b)
    for l in (1.5, 0.2, 0.001):
        h = HODLR_Matrix(n, n, KernelSpec(kind, l, 0.25), P, 64)
        torch.cuda.synchronize()
        h.kernel_matvec_device(b.data_ptr(), y.data_ptr(), nrhs)
        torch.cuda.synchronize()
        K, x = _reference(kind, dim, l, P, cols, 0.25)
        err = np.abs(y.cpu().numpy().T - K).astype(float)
        bound = _bound(kind, dim, l, P, K, x)
        assert np.all(err <= bound), (l, float((err / bound).max()))
