"""The work a program gives this framework, as cases that can be timed and checked.

A case is a dict of plain values.  `listed()` names twelve of them, `draw(rng)`
gives more of the same ranges, `prepare` builds what a program has in hand
before the call, `run` is one pass through the public entry points, `work` what
the pass cannot do without, and `exact` the same results in 64 bits from plain
torch.

Solves run a fixed number of iterations (as the drop-in entry points do) except
where a case has a tolerance, so two builds of the library return the same
iterate.  Coefficients vary by a few per cent for the same reason: what a kernel
does depends on the pattern, but the rounding of an iterate is amplified by the
outlying eigenvalues of strongly varying ones.  Matrices are the repository's own workloads: constant and variable
coefficient stencils in 2D and 3D, upwind convection-diffusion, 27-point
systems, and an irregular graph matrix like the circuit matrices the reference
is measured on.  Grids are drawn with any side, so row counts need not be
multiples of the 16-row tile.
"""
from __future__ import annotations

import itertools
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mille-feuille_b200"))

import millefeuille as mf  # noqa: E402
from millefeuille.autograd import SolvePattern, sparse_solve  # noqa: E402

DEV = "cuda:0"


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # a product with a small operator: one call inside somebody's loop, all latency
        dict(name="spmv_small", kind="spmv", grid="lap2", nx=97, ny=96, nz=1, prec="fp64", noalloc=False),
        # the same on a large 3D system: the matrix is streamed from memory
        dict(name="spmv_large", kind="spmv", grid="var3", nx=128, ny=128, nz=128, prec="fp64", noalloc=False),
        # the smallest solve in the benchmark: 2D Laplacian to 1e-10, bound by its grid syncs
        dict(name="cg_lap256_tol", kind="solve", grid="lap2", nx=256, ny=256, nz=1, method="cg", prec="fp64",
             iters=10000, tol=1e-10, host=False),
        # the headline system, mixed precision, two residual replacements
        dict(name="cg_var128_mixed", kind="solve", grid="var3", nx=128, ny=128, nz=128, method="cg", prec="mixed",
             iters=100, tol=0.0, host=False),
        # vectors larger than the L2 cache: everything streams, values exact in FP16
        dict(name="cg_lap2048_mixed", kind="solve", grid="lap2", nx=2048, ny=2048, nz=1, method="cg", prec="mixed",
             iters=100, tol=0.0, host=False),
        # an irregular matrix handed over in host arrays, row count not a multiple of 16
        dict(name="cg_graph_host", kind="solve", grid="graph", nx=60013, ny=1, nz=1, method="cg", prec="fp64",
             iters=40, tol=0.0, host=True),
        # nonsymmetric convection-diffusion
        dict(name="bicgstab_conv96", kind="solve", grid="conv3", nx=96, ny=96, nz=96, method="bicgstab", prec="fp64",
             iters=20, tol=0.0, host=False),
        # eight right-hand sides of the 2D anisotropic system in one launch
        dict(name="multi8_aniso512", kind="multi", grid="var2", nx=512, ny=512, nz=1, prec="mixed", iters=100, nrhs=8),
        # many small systems of uneven size, each with its own right-hand sides
        dict(name="batch_uneven", kind="batch", systems=40, prec="mixed", iters=40, cap=4, lo2=32, hi2=256, lo3=8,
             hi3=32),
        # a training step on the coefficients: new values, forward, adjoint, gradients
        dict(name="train_cg", kind="train", grid="var2", nx=256, ny=255, nz=1, method="cg", prec="mixed", iters=60,
             nrhs=4),
        # the same for a nonsymmetric operator, whose adjoint needs the transposed handle
        dict(name="train_bicgstab", kind="train", grid="conv3", nx=48, ny=47, nz=49, method="bicgstab", prec="fp64",
             iters=20, nrhs=1),
        # a new matrix every time step: tiling and encoding on the GPU, then one product
        dict(name="build_var96", kind="build", grid="var3", nx=96, ny=96, nz=96, prec="fp64"),
    ]


GRIDS = {"lap2": (2, 5), "var2": (2, 5), "var3": (3, 7), "conv3": (3, 7), "st27": (3, 27), "graph": (1, 11)}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, names, lo, hi):
    """A grid of about lo..hi unknowns (log-uniform), sides uneven."""
    g = rng.choice(names)
    n = _log(rng, lo, hi)
    dim = GRIDS[g][0]
    if dim == 1:
        return dict(grid=g, nx=n, ny=1, nz=1)
    s = n ** (1.0 / dim)
    nx = max(2, int(s * math.exp(rng.uniform(-0.5, 0.0))))
    ny = max(2, int(s * math.exp(rng.uniform(-0.5, 0.0))))
    nz = max(2, int(s)) if dim == 3 else 1
    return dict(grid=g, nx=nx, ny=ny, nz=nz)


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "solve", "solve", "solve", "solve", "multi", "batch", "train", "build"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "spmv":
        c = _grid(rng, ["lap2", "var2", "var3", "st27", "graph"], 300, 2_500_000)
        if c["grid"] in ("st27", "graph"):
            c["nx"] = max(2, c["nx"] // 4)
        n = c["nx"] * c["ny"] * c["nz"]                   # the allocation-free call takes up to 2^21 entries
        return dict(kind=kind, prec=prec, noalloc=n < 2_000_000 and rng.random() < 0.5, **c)
    if kind == "solve":
        method = rng.choice(["cg", "cg", "bicgstab"])
        names = ["lap2", "var2", "var3", "st27", "graph"] if method == "cg" else ["conv3", "var3"]
        c = _grid(rng, names, 1000, 4_000_000 if method == "cg" else 1_000_000)
        if c["grid"] in ("st27", "graph"):
            c["nx"] = max(2, c["nx"] // 6)
        n = c["nx"] * c["ny"] * c["nz"]
        # short of full convergence, where nothing is left to iterate on
        iters = min(rng.randint(20, 120), int(1.2 * n ** 0.5)) if method == "cg" else min(rng.randint(8, 16),
                                                                                          int(n ** (1 / 3)))
        if c["grid"] in ("st27", "graph"):
            iters = min(iters, 30)
        return dict(kind=kind, method=method, prec=prec, iters=iters, tol=0.0, host=n < 500_000 and rng.random() < 0.3,
                    **c)
    if kind == "multi":
        return dict(kind=kind, prec=prec, iters=rng.randint(20, 80), nrhs=rng.randint(2, 8),
                    **_grid(rng, ["var2", "var3"], 1000, 260_000))
    if kind == "batch":
        lo2, lo3 = rng.randint(16, 48), rng.randint(5, 10)
        return dict(kind=kind, systems=rng.randint(4, 40), prec=prec, iters=rng.randint(10, 40),
                    cap=rng.choice([1, 2, 4, 8]), lo2=lo2, hi2=rng.randint(lo2 + 8, 256), lo3=lo3,
                    hi3=rng.randint(lo3 + 2, 32))
    if kind == "train":
        method = rng.choice(["cg", "bicgstab"])
        return dict(kind=kind, method=method, prec=prec, iters=rng.randint(20, 60) if method == "cg" else 12,
                    nrhs=rng.randint(1, 8) if method == "cg" else rng.randint(1, 2),
                    **_grid(rng, ["var2", "var3"] if method == "cg" else ["conv3"], 2000, 110_000))
    return dict(kind=kind, prec=prec, **_grid(rng, ["lap2", "var2", "var3", "st27"], 1000, 300_000))


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 1000003 + 17)


def _normal(gen, *shape):
    return torch.randn(*shape, generator=gen, device=DEV, dtype=torch.float64)


def _uniform(gen, *shape):
    return torch.rand(*shape, generator=gen, device=DEV, dtype=torch.float64) * 2 - 1


def _csr(n, rows, cols, vals):
    """CSR (int32 pointers and columns) from unique coordinate entries."""
    order = torch.argsort(rows * n + cols)
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    rowptr[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return rowptr.to(torch.int32), cols[order].to(torch.int32), vals[order].contiguous()


def _stencil(case, gen):
    """Grid operators, x fastest: one coefficient per pair of neighbours, Dirichlet
    boundary (a missing neighbour leaves its coefficient on the diagonal)."""
    g = case["grid"]
    dim = GRIDS[g][0]
    shape = (case["nz"], case["ny"], case["nx"]) if dim == 3 else (1, case["ny"], case["nx"])
    n = shape[0] * shape[1] * shape[2]
    lin = torch.arange(n, device=DEV).reshape(shape)
    axes = [(0, 0, 1), (0, 1, 0), (1, 0, 0)][:dim]
    dirs = axes if g != "st27" else [d for d in itertools.product((-1, 0, 1), repeat=3) if d > (0, 0, 0)]
    diag = torch.zeros(n, dtype=torch.float64, device=DEV)
    rows, cols, vals = [], [], []
    grid_pos = torch.meshgrid(*[torch.arange(s, device=DEV) for s in shape], indexing="ij")
    for d in dirs:
        lo = tuple(slice(max(0, -s), shape[a] - max(0, s)) for a, s in enumerate(d))
        hi = tuple(slice(max(0, s), shape[a] - max(0, -s)) for a, s in enumerate(d))
        i, j = lin[lo].reshape(-1), lin[hi].reshape(-1)
        base = 1.0
        if g == "lap2":
            e = f = torch.ones(i.numel(), dtype=torch.float64, device=DEV)
        elif g == "conv3":
            # first-order upwind: the flow enters through one of the two neighbours
            h = 2 * math.pi / max(shape)
            a = axes.index(d)
            v = 10.0 * h * torch.sin((grid_pos[(1, 0, 2)[a]][lo].reshape(-1).double() + 0.5) * h)
            e, f = 1 + torch.clamp(-v, min=0), 1 + torch.clamp(v, min=0)
        else:
            sigma = 0.5 if g == "st27" else 0.05
            base = 10.0 if g == "var2" and d == (0, 0, 1) else 1.0
            e = f = base * torch.exp(sigma * _normal(gen, i.numel()))
        rows += [i, j]
        cols += [j, i]
        vals += [-e, -f]
        diag.index_add_(0, i, e)
        diag.index_add_(0, j, f)
        inside = torch.zeros(n, dtype=torch.float64, device=DEV)
        inside.index_add_(0, i, torch.ones_like(e))
        inside.index_add_(0, j, torch.ones_like(e))
        diag += base * (2 - inside)
    rows.append(lin.reshape(-1))
    cols.append(lin.reshape(-1))
    vals.append(diag)
    return n, *_csr(n, torch.cat(rows), torch.cat(cols), torch.cat(vals))


def _graph(case, gen):
    """A weighted graph Laplacian plus a small diagonal: most neighbours near, some anywhere."""
    n = case["nx"]
    i = torch.arange(n, device=DEV).repeat(5)
    near = i + (_normal(gen, 5 * n) * 40).round().long()
    far = torch.randint(0, n, (5 * n,), generator=gen, device=DEV)
    j = torch.where(torch.rand(5 * n, generator=gen, device=DEV) < 0.1, far, near).remainder(n)
    key = torch.unique(torch.minimum(i, j) * n + torch.maximum(i, j))
    i, j = key // n, key % n
    i, j = i[i != j], j[i != j]
    w = torch.exp(0.3 * _normal(gen, i.numel()))
    rowptr, cols, vals = _csr(n, torch.cat([i, j]), torch.cat([j, i]), torch.cat([w, w]))
    diag = 0.05 + torch.segment_reduce(vals, "sum", offsets=rowptr.long())
    k = torch.arange(n, device=DEV)
    return n, *_csr(n, torch.cat([i, j, k]), torch.cat([j, i, k]), torch.cat([-w, -w, diag]))


def _matrix(case, gen):
    return _graph(case, gen) if case["grid"] == "graph" else _stencil(case, gen)


def _sparse(n, rowptr, colidx, val):
    return torch.sparse_csr_tensor(rowptr.long(), colidx.long(), val, size=(n, n))


def _batch_cases(case):
    """The systems of a batch: alternately 2D 5-point and 3D 27-point, sides spread over their ranges."""
    out = []
    for k in range(case["systems"]):
        t = ((k * 7) % case["systems"]) / max(1, case["systems"] - 1)
        if k % 2:
            s = int(round(case["lo3"] + t * (case["hi3"] - case["lo3"])))
            out.append((dict(grid="st27", nx=s, ny=s, nz=s), 1 + k % 5))
        else:
            s = int(round(case["lo2"] + t * (case["hi2"] - case["lo2"])))
            out.append((dict(grid="var2", nx=s, ny=s, nz=1), 1 + k % 5))
    return out


def _inputs(case, seed):
    """Everything random in a case, from the seed alone."""
    gen = _gen(seed)
    kind = case["kind"]
    if kind == "batch":
        out = []
        for c, nrhs in _batch_cases(case):
            A = _matrix(c, gen)
            out.append((A, _normal(gen, nrhs, A[0])))
        return out
    A = _matrix(case, gen)
    n = A[0]
    if kind in ("spmv", "build"):
        return A, _uniform(gen, n)
    if kind == "solve":
        rowptr, colidx, val = A[1:]
        x = _uniform(gen, n)
        return A, torch.segment_reduce(val * x[colidx.long()], "sum", offsets=rowptr.long())       # b = A x
    if kind == "multi":
        return A, _normal(gen, case["nrhs"], n)
    return A, _normal(gen, case["nrhs"], n), _normal(gen, case["nrhs"], n)


def _options(case):
    return mf.default_options(method=case.get("method", "cg"), precision=case["prec"], tol=case.get("tol", 0.0),
                              max_iter=case["iters"], fixed_iters=0 if case.get("tol", 0.0) > 0 else 1)


def prepare(case, seed):
    kind = case["kind"]
    got = _inputs(case, seed)
    st = {"case": case}
    if kind == "batch":
        st["mats"] = [mf.Matrix.from_csr(A[0], A[0], *A[1:]) for A, _ in got]
        st["B"] = [B for _, B in got]
        st["X"] = [torch.zeros_like(B) for B in st["B"]]
        st["batch"] = mf.Batch(st["mats"], [B.shape[0] for B in st["B"]])
        st["batch"].configure(case["cap"], 1)
        st["opts"] = _options(case)
        return st
    n, rowptr, colidx, val = got[0]
    if kind in ("spmv", "solve", "multi"):
        st["A"] = mf.Matrix.from_csr(n, n, rowptr, colidx, val)
        st["v"] = got[1].cpu().numpy() if case.get("host") else got[1]
        if kind == "spmv":
            st["y"] = torch.zeros(n, dtype=torch.float64, device=DEV)
        else:
            st["opts"] = _options(case)
    elif kind == "build":
        st.update(n=n, csr=(rowptr, colidx, val), v=got[1])
    else:
        st.update(csr=(rowptr, colidx), new_val=val, val=val.clone().requires_grad_(),
                  b=got[1].clone().requires_grad_(), target=got[2],
                  pattern=SolvePattern(rowptr, colidx, n, symmetric=case["method"] == "cg"))
    return st


# ---------------------------------------------------------------- one pass
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "spmv":
        if case["noalloc"]:
            return st["A"].spmv_noalloc(st["v"], st["y"], precision=case["prec"])
        return st["A"].spmv(st["v"], precision=case["prec"])
    if kind == "solve":
        return st["A"].solve(st["v"], options=st["opts"])[0]
    if kind == "multi":
        return st["A"].solve_multi(st["v"], options=st["opts"])[0]
    if kind == "batch":
        return st["batch"].solve(st["B"], st["X"], options=st["opts"])[0]
    if kind == "build":
        return mf.Matrix.from_csr(st["n"], st["n"], *st["csr"]).spmv(st["v"], precision=case["prec"])
    with torch.no_grad():
        st["val"].copy_(st["new_val"])        # this step's coefficients, in the program's own buffer
    st["val"].grad = st["b"].grad = None
    x = sparse_solve(*st["csr"], st["val"], st["b"], method=case["method"], precision=case["prec"], tol=0.0,
                     pattern=st["pattern"], max_iter=case["iters"], fixed_iters=1)
    (x - st["target"]).square().sum().backward()
    return x.detach(), st["val"].grad, st["b"].grad


# ---------------------------------------------------------------- what it cannot do without
def _size(c):
    n = c["nx"] * c["ny"] * c["nz"]
    if c["grid"] == "graph":
        return n, 11 * n
    sides = [c["nx"], c["ny"], c["nz"]][:GRIDS[c["grid"]][0]]
    if c["grid"] == "st27":
        return n, math.prod(3 * s - 2 for s in sides)
    return n, n + sum(2 * n // s * (s - 1) for s in sides)


def _solve_work(n, nnz, iters, nrhs, bicg, value_bytes):
    """Per iteration: each product reads the values and a byte of index per entry, and each
    vector of the method is read and written once (CG: x r p q; BiCGSTAB: x r p v s t, and the shadow residual)."""
    products, vectors = (2, 104) if bicg else (1, 64)
    return dict(bytes=iters * (products * nnz * (value_bytes + 1.0) + vectors * n * nrhs),
                flops=iters * nrhs * (products * 2.0 * nnz + (24.0 if bicg else 12.0) * n))


def work(case):
    kind = case["kind"]
    vb = 8 if case["prec"] == "fp64" else 4
    if kind == "batch":
        parts = [_solve_work(*_size(c), case["iters"], nrhs, False, vb) for c, nrhs in _batch_cases(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n, nnz = _size(case)
    if case["grid"] == "lap2" and kind == "solve" and vb == 4:
        vb = 2                                   # every value is exact in FP16
    if kind == "spmv":
        return dict(bytes=nnz * (vb + 1.0) + 16.0 * n, flops=2.0 * nnz)
    if kind == "build":
        # the CSR read; the tile layout and the slices written (every stored precision), read back once
        return dict(bytes=12.0 * nnz + 4.0 * n + 2 * 17.0 * nnz + nnz * (vb + 1.0) + 16.0 * n, flops=2.0 * nnz)
    if kind == "train":
        w = _solve_work(n, nnz, 2 * case["iters"], case["nrhs"], case["method"] == "bicgstab", vb)
        return dict(bytes=w["bytes"] + 46.0 * nnz + 8.0 * nnz + 16.0 * n * case["nrhs"],
                    flops=w["flops"] + 2.0 * nnz * case["nrhs"])
    iters = min(case["iters"], 3 * max(case["nx"], case["ny"]))     # to a tolerance: about that many
    return _solve_work(n, nnz, iters, case.get("nrhs", 1), case.get("method") == "bicgstab", vb)


# ---------------------------------------------------------------- the same in 64 bits
def _cg(S, b, iters, tol):
    x, r = torch.zeros_like(b), b.clone()
    p, rr = r.clone(), (r * r).sum()
    stop = tol * tol * rr
    for _ in range(iters):
        q = S @ p
        alpha = rr / (p * q).sum()
        x += alpha * p
        r -= alpha * q
        new = (r * r).sum()
        if tol > 0 and new <= stop:
            break
        p = r + (new / rr) * p
        rr = new
    return x


def _bicgstab(S, b, iters, tol):
    x, r, rh, p = torch.zeros_like(b), b.clone(), b.clone(), b.clone()
    rho = (rh * r).sum()
    for _ in range(iters):
        v = S @ p
        alpha = rho / (rh * v).sum()
        s = r - alpha * v
        t = S @ s
        omega = (t * s).sum() / (t * t).sum()
        x += alpha * p + omega * s
        r = s - omega * t
        new = (rh * r).sum()
        p = r + (new * alpha) / (rho * omega) * (p - omega * v)
        rho = new
    return x


def exact(case, seed):
    kind = case["kind"]
    got = _inputs(case, seed)
    solver = _bicgstab if case.get("method") == "bicgstab" else _cg

    def columns(S, B):
        return torch.stack([solver(S, b, case["iters"], case.get("tol", 0.0)) for b in B])

    if kind == "batch":
        return [columns(_sparse(*A), B) for A, B in got]
    A = got[0]
    S = _sparse(*A)
    if kind in ("spmv", "build"):
        return S @ got[1]
    if kind == "solve":
        x = solver(S, got[1], case["iters"], case["tol"])
        return x.cpu().numpy() if case["host"] else x
    if kind == "multi":
        return columns(S, got[1])
    n, rowptr, colidx, val = A
    X = columns(S, got[1])
    G = 2 * (X - got[2])
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), (rowptr[1:] - rowptr[:-1]).long())
    lam = columns(_sparse(n, *_csr(n, colidx.long(), rows, val)), G)       # the transposed system
    grad = torch.zeros_like(val)
    for k in range(X.shape[0]):
        grad -= lam[k][rows] * X[k][colidx.long()]
    return X, grad, lam
