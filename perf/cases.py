"""What the performance of this solver is judged by: the calls that its users make.

Each case is one of
  fit      a new system: points (or a dense matrix) and right-hand sides in host
           memory, HODLR_Matrix built, compressed, factored and solved once
           (recLU_Solve) -- one evaluation of a model's hyperparameters;
  krylov   a new system solved to ||b - K x|| / ||b|| <= 1e-10 by HODLR-
           preconditioned GMRES (iterative_Solve) -- ACA, factorization, direct
           solves and full-kernel products in the proportions of real use;
  solve    more right-hand sides for a system factored before (device buffers);
  product  the full-kernel product K X (device buffers), the residual check of
           every refinement;
  forest   many small systems of uneven size in one handle, refined to 1e-10.

Sizes, kernels, length scales and tolerances are those of the repository's
configurations, tests and benchmark (bench.py, tests/), or lie between them.
"""
import math
import random

import numpy as np
import torch

from dense_hodlr_b200 import HODLR_Matrix, KernelSpec


def listed():
    return [
        # the smallest calls: the smoke test's system, and the 1D Gaussian
        # configuration (N = 4096); launches and waits are all there is
        dict(name="fit_1d_1024", do="fit", n=1024, dim=1, cloud="uniform", kernel="gaussian",
             l=0.1, shift=1.0, leaf=64, tol=1e-10, nrhs=2),
        dict(name="fit_1d_4096", do="fit", n=4096, dim=1, cloud="uniform", kernel="gaussian",
             l=0.1, shift=1.0, leaf=64, tol=1e-10, nrhs=1),
        # a matrix given entry by entry, with the default leaf size (uneven leaves)
        dict(name="fit_dense_2001", do="fit", n=2001, dim=1, cloud="dense",
             kernel="inv_multiquadric", l=0.15, shift=0.5, leaf=30, tol=1e-8, nrhs=1),
        # an ordinary 2D system of an odd size
        dict(name="fit_2d_20011", do="fit", n=20011, dim=2, cloud="uniform", kernel="matern32",
             l=0.2, shift=1e-1, leaf=128, tol=1e-8, nrhs=4),
        # high ranks: points on a sphere at a tight tolerance
        dict(name="krylov_sphere_16384", do="krylov", n=16384, dim=3, cloud="sphere",
             kernel="matern32", l=0.1, shift=1e-2, leaf=128, tol=1e-10, nrhs=1,
             precision="fp64"),
        # the mixed-precision form: Woodbury products in 3xTF32, 16 right-hand sides
        dict(name="krylov_tf32x3_cube_40000", do="krylov", n=40000, dim=3, cloud="uniform",
             kernel="gaussian", l=0.3, shift=1e-1, leaf=128, tol=1e-8, nrhs=16,
             precision="tf32x3"),
        # the benchmark's configuration: the largest whole call
        dict(name="krylov_2d_262144", do="krylov", n=262144, dim=2, cloud="uniform",
             kernel="matern32", l=0.2, shift=1e-2, leaf=128, tol=1e-8, nrhs=8,
             precision="fp64"),
        # more right-hand sides for a factored system, one and several at a time
        dict(name="solve_2d_30001_x1", do="solve", n=30001, dim=2, cloud="uniform",
             kernel="matern32", l=0.2, shift=1e-1, leaf=128, tol=1e-8, nrhs=1),
        dict(name="solve_2d_262144_x8", do="solve", n=262144, dim=2, cloud="uniform",
             kernel="matern32", l=0.2, shift=1e-2, leaf=128, tol=1e-8, nrhs=8),
        # the full-kernel product, one vector of an odd 3D cloud and a panel in 2D
        dict(name="product_3d_50001_x1", do="product", n=50001, dim=3, cloud="uniform",
             kernel="gaussian", l=0.3, shift=1e-1, nrhs=1),
        dict(name="product_2d_131072_x8", do="product", n=131072, dim=2, cloud="uniform",
             kernel="matern32", l=0.2, shift=1e-2, nrhs=8),
        # uneven independent systems in one handle (1D / 2D, Gaussian / Matern-3/2)
        dict(name="forest_40", do="forest", systems=40, n_min=1024, n_max=8192, mix=11, leaf=64,
             tol=1e-8, nrhs=1),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    do = rng.choice(["fit", "fit", "krylov", "solve", "product", "forest"])
    if do == "forest":
        lo = int(_log_uniform(rng, 512, 2048))
        return dict(do="forest", systems=rng.randrange(4, 41), n_min=lo,
                    n_max=int(lo * rng.uniform(1.5, 8.0)) + 1, mix=rng.randrange(1 << 20),
                    leaf=rng.choice([32, 64, 100]), tol=1e-8, nrhs=rng.choice([1, 2, 3]))
    if do == "product":
        return dict(do="product", n=int(_log_uniform(rng, 1000, 131072)), dim=rng.choice([1, 2, 3]),
                    cloud="uniform",
                    kernel=rng.choice(["gaussian", "matern32", "inv_multiquadric", "exponential",
                                       "quadratic"]),
                    l=round(_log_uniform(rng, 0.05, 0.5), 4), shift=round(_log_uniform(rng, 1e-2, 1.0), 4),
                    nrhs=rng.choice([1, 2, 4, 5, 8, 11, 16]))
    dim = rng.choice([1, 1, 2, 2, 2, 3])
    hi = {"fit": (20000, 60000, 12000), "krylov": (30000, 100000, 16000),
          "solve": (60000, 200000, 20000)}[do][dim - 1]
    cloud, l = "uniform", round(_log_uniform(rng, 0.1, 0.5), 4)
    kernel = rng.choice(["gaussian", "matern32", "inv_multiquadric"])
    if dim == 3:
        l = round(rng.uniform(0.3, 0.5), 4)
        cloud = rng.choice(["uniform", "sphere"]) if do == "krylov" else "uniform"
        kernel = "gaussian" if cloud == "uniform" else "matern32"
    n = int(_log_uniform(rng, 600, hi))
    case = dict(do=do, n=n, dim=dim, cloud=cloud, kernel=kernel, l=l,
                shift=round(_log_uniform(rng, 1e-1, 1.0), 4), leaf=rng.choice([30, 64, 100, 128]),
                tol=rng.choice([1e-6, 1e-8, 1e-8, 1e-10] if dim < 3 else [1e-6, 1e-8]),
                nrhs=rng.choice([1, 2, 3, 8, 16]))
    if do == "fit" and dim == 1 and n <= 3000 and rng.random() < 0.5:
        case["cloud"] = "dense"
    if do == "krylov":
        case["precision"] = rng.choice(["fp64", "fp64", "tf32x3"])
    return case


# ------------------------------------------------------------------ inputs
def _kd_sorted(pts, smallest=8):
    """k-d median order of dim x n points (left part floor(n / 2)), down to small clusters."""
    dim, n = pts.shape
    sizes = torch.tensor([n], device=pts.device)
    depth = 0
    while int(sizes.max()) > smallest:
        seg = torch.repeat_interleave(torch.arange(len(sizes), device=pts.device), sizes)
        by_key = torch.argsort(pts[depth % dim], stable=True)
        order = by_key[torch.argsort(seg[by_key], stable=True)]
        pts = pts[:, order]
        left = sizes // 2
        sizes = torch.stack([left, sizes - left], 1).reshape(-1)
        depth += 1
    return pts.contiguous()


def _points(n, dim, cloud, gen):
    if dim == 1:
        p = torch.rand(1, n, dtype=torch.float64, device="cuda", generator=gen) * 2.0 - 1.0
        return torch.sort(p, dim=1).values
    if cloud == "sphere":
        p = torch.randn(dim, n, dtype=torch.float64, device="cuda", generator=gen)
        p = p / p.norm(dim=0, keepdim=True)
    else:
        p = torch.rand(dim, n, dtype=torch.float64, device="cuda", generator=gen)
    return _kd_sorted(p)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rhs(n, nrhs, gen):
    """nrhs x n on the device: row c is column c of a column-major n x nrhs panel."""
    return torch.randn(nrhs, n, dtype=torch.float64, device="cuda", generator=gen)


def _systems(case):
    """(n, dim, kernel, l, shift) of a forest's systems."""
    rng = random.Random(case["mix"])
    return [(int(_log_uniform(rng, case["n_min"], case["n_max"])), rng.choice([1, 2]),
             rng.choice(["gaussian", "matern32"]), _log_uniform(rng, 0.05, 0.5),
             _log_uniform(rng, 1e-1, 1.0)) for _ in range(case["systems"])]


def _entries(kernel, l, shift, x, y, row0=None):
    """K(x, y) for dim x n points, in 64 bits; the shift where row0 + i == j."""
    r2 = torch.zeros(x.shape[1], y.shape[1], dtype=torch.float64, device=x.device)
    for d in range(x.shape[0]):
        r2 += (x[d][:, None] - y[d][None, :]) ** 2
    if kernel == "gaussian":
        k = torch.exp(r2.mul_(-1.0 / (l * l)))
    elif kernel == "matern32":
        s = r2.sqrt_().mul_(math.sqrt(3.0) / l)
        k = torch.exp(-s).mul_(s.add_(1.0))
    elif kernel == "inv_multiquadric":
        k = torch.rsqrt(r2.mul_(1.0 / (l * l)).add_(1.0))
    elif kernel == "exponential":
        k = torch.exp(r2.sqrt_().mul_(-1.0 / l))
    else:  # quadratic
        k = r2.mul_(1.0 / (l * l)).add_(1.0)
    if row0 is not None:
        i = torch.arange(x.shape[1], device=x.device)
        k[i, row0 + i] += shift
    return k


def _inputs(case, seed):
    gen = _generator(seed)
    if case["do"] == "forest":
        pts = [_points(n, dim, "uniform", gen) for n, dim, _, _, _ in _systems(case)]
        return pts, _rhs(sum(p.shape[1] for p in pts), case["nrhs"], gen)
    pts = _points(case["n"], case["dim"], case["cloud"], gen)
    return pts, _rhs(case["n"], case["nrhs"], gen)


def _spec(case):
    return KernelSpec(case["kernel"], case["l"], case["shift"])


def _matrix(case, pts):
    """A new system from host memory, as a user's program builds it."""
    n = case["n"]
    if case["cloud"] == "dense":
        h = HODLR_Matrix(pts, case["leaf"])
    else:
        h = HODLR_Matrix(n, n, _spec(case), pts, case["leaf"])
    h.set_LRTolerance(case["tol"])
    return h


def prepare(case, seed):
    pts, b = _inputs(case, seed)
    if case["do"] == "forest":
        systems = [(p.cpu().numpy(), KernelSpec(kind, l, shift))
                   for p, (_, _, kind, l, shift) in zip(pts, _systems(case))]
        return dict(case=case, systems=systems, b=b, x=torch.empty_like(b))
    if case["do"] in ("fit", "krylov"):
        host = (_entries(case["kernel"], case["l"], case["shift"], pts, pts, 0)
                if case["cloud"] == "dense" else pts).cpu().numpy()
        return dict(case=case, pts=host, b=np.asfortranarray(b.cpu().numpy().T))
    leaf = case.get("leaf", 128)
    h = HODLR_Matrix(case["n"], case["n"], _spec(case), pts.cpu().numpy(), leaf)
    if case["do"] == "solve":
        h.set_LRTolerance(case["tol"])
        h.recLU_Compute()
    torch.cuda.synchronize()  # b is ready before another stream reads it
    return dict(case=case, h=h, b=b, x=torch.empty_like(b))


def run(state):
    case = state["case"]
    do = case["do"]
    if do == "fit":
        return _matrix(case, state["pts"]).recLU_Solve(state["b"])
    if do == "krylov":
        h = _matrix(case, state["pts"])
        h.set_precision(case["precision"])
        return h.iterative_Solve(state["b"], maxIterations=200, stop_tolerance=1e-10)
    b, x = state["b"], state["x"]
    if do == "forest":
        h = HODLR_Matrix.forest(state["systems"], case["leaf"])
        h.set_LRTolerance(case["tol"])
        h.forest_refine_device(b.data_ptr(), x.data_ptr(), case["nrhs"], tol=1e-10)
    elif do == "solve":
        state["h"].solve_device(b.data_ptr(), x.data_ptr(), case["nrhs"])
    else:
        state["h"].kernel_matvec_device(b.data_ptr(), x.data_ptr(), case["nrhs"])
    return x


# --------------------------------------------------------- floors and values
def _rank(case):
    """A block's rank, roughly: what ACA finds at the top of such a cloud."""
    n, dim = case["n"], case["dim"]
    digits = -math.log10(case["tol"])
    if dim == 1:
        return 2.0 * digits
    if case["cloud"] == "sphere":
        return min(n / 4, 0.8 * digits * math.sqrt(n) / 1.3)
    return (12.0 if dim == 2 else 40.0) * digits * (1.0 + 0.1 * math.log2(n / 1024.0))


def _one(n, nrhs, leaf, rank, dim):
    """(bytes, flops) of compressing and factoring one system, and of one direct solve.

    Compression evaluates and writes rank columns of W and V per level and updates
    each by the earlier ones; the factorization turns the U panels into K^-1 U
    (per level a product with, and an update of, the columns of all levels above);
    a solve reads V, K^-1 U and the leaf factors once.
    """
    levels = max(1, math.ceil(math.log2(max(2.0, n / leaf))))
    cols = [min(rank * 2.0 ** (-0.4 * k), n / 2.0 ** (k + 1)) for k in range(levels)]
    total = sum(cols)
    comp = (16.0 * n * total + 8.0 * n * dim, sum(2.0 * 2.0 * n * k * k for k in cols))
    above, fact_flops = 0.0, 2.0 / 3.0 * n * leaf * leaf + 2.0 * n * leaf * total
    for k in cols:
        fact_flops += 2.0 * n * k * (above + k) + 2.0 * n * k * above
        above += k
    fact = (24.0 * n * total + 8.0 * n * leaf, fact_flops)
    sol = (8.0 * n * (2.0 * total + leaf + 2.0 * nrhs), 2.0 * n * nrhs * (2.0 * total + leaf))
    return comp, fact, sol


def _product_flops(n, nrhs):
    """One entry is evaluated for a pair of points and used in both directions."""
    return 0.5 * n * n * (33.0 + 4.0 * nrhs)


def work(case):
    do = case["do"]
    if do == "product":
        n, q = case["n"], case["nrhs"]
        return {"bytes": 8.0 * n * (case["dim"] + 2 * q), "flops": _product_flops(n, q)}
    if do == "forest":
        nbytes = flops = 0.0
        for n, dim, _, _, _ in _systems(case):
            c, f, s = _one(n, case["nrhs"], case["leaf"],
                           _rank(dict(n=n, dim=dim, tol=case["tol"], cloud="uniform")), dim)
            nbytes += c[0] + f[0] + 3 * s[0]
            flops += c[1] + f[1] + 3 * s[1] + 3 * _product_flops(n, case["nrhs"])
        return {"bytes": nbytes, "flops": flops}
    c, f, s = _one(case["n"], case["nrhs"], case["leaf"], _rank(case), case["dim"])
    if do == "solve":
        return {"bytes": s[0], "flops": s[1]}
    if do == "fit":
        extra = 8.0 * case["n"] ** 2 if case["cloud"] == "dense" else 0.0
        return {"bytes": c[0] + f[0] + s[0] + extra, "flops": c[1] + f[1] + s[1]}
    # krylov: the direct solve and at least two iterations
    return {"bytes": c[0] + f[0] + 3 * s[0],
            "flops": c[1] + f[1] + 3 * s[1] + 3 * _product_flops(case["n"], case["nrhs"])}


def _dense_solve(k, b):
    """K^-1 b for b nrhs x n, with one step of refinement."""
    c = torch.linalg.cholesky(k)
    x = torch.cholesky_solve(b.T, c)
    x += torch.cholesky_solve(b.T - k @ x, c)
    return x


def exact(case, seed):
    if case["do"] == "forest":
        pts, b = _inputs(case, seed)
        out, o = torch.empty_like(b), 0
        for p, (n, _, kind, l, shift) in zip(pts, _systems(case)):
            out[:, o:o + n] = _dense_solve(_entries(kind, l, shift, p, p, 0), b[:, o:o + n]).T
            o += n
        return out
    if case["do"] == "product":
        pts, b = _inputs(case, seed)
        out = torch.empty_like(b)
        for r0 in range(0, case["n"], 4096):
            k = _entries(case["kernel"], case["l"], case["shift"], pts[:, r0:r0 + 4096], pts, r0)
            out[:, r0:r0 + 4096] = (k @ b.T).T
        return out
    if case["n"] > 33000:
        return None
    pts, b = _inputs(case, seed)
    x = _dense_solve(_entries(case["kernel"], case["l"], case["shift"], pts, pts, 0), b)
    return x.T.contiguous() if case["do"] == "solve" else x.cpu().numpy()
