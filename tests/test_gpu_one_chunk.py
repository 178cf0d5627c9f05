"""Matrices whose every tile-row is one chunk (rows of up to 8 entries in up to 15
tiles) have walks and solve kernels of their own, by their longest row (5, 7, 8).
Row counts at the edges of a tile-row (16), of a block's turn (32 tile-rows), of
one cluster (512 tile-rows), of one and two blocks per SM (where CG iterations
stop being kept in registers); longest rows on both sides of each kernel's limit; a matrix with
one empty tile-row (which takes the general kernels) beside each.

Bounds: a product's row is a sum of k <= 9 terms in FP64, within k eps of
sum |a||x| (k + 1 here); an FP32-stored one adds 2^-24 of it.  Three CG or
BiCGSTAB iterations on these matrices (diagonally dominant, condition below 10)
amplify rounding by less than 1e4."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _banded(n, longest, seed, empty_tile_row=False):
    """Symmetric, diagonally dominant, `longest` entries in the longest row."""
    rng = np.random.default_rng(seed)
    half = [1, 17, 40][: (longest - 1) // 2]
    S = sp.lil_matrix((n, n))
    for o in half:
        if o < n:
            v = rng.uniform(0.5, 1.0, n - o)
            S = S + sp.diags([-v, -v], [o, -o])
    S = sp.csr_matrix(S)
    if longest % 2 == 0 and n > 60:                 # one more pair, in two rows only
        E = sp.lil_matrix((n, n))
        E[20, 55] = E[55, 20] = -0.25
        S = S + sp.csr_matrix(E)
    if empty_tile_row and n > 64:
        keep = np.ones(n)
        keep[32:48] = 0.0
        S = sp.diags(keep) @ S @ sp.diags(keep)
    d = np.asarray(abs(S).sum(axis=1)).ravel() + rng.uniform(1.0, 2.0, n)
    if empty_tile_row and n > 64:
        d[32:48] = 0.0
    A = sp.csr_matrix(S + sp.diags(d))
    A.eliminate_zeros()
    A.sort_indices()
    return A


def _cg(A, b, k):
    x, r = np.zeros_like(b), b.copy()
    p, rr = r.copy(), r @ r
    for _ in range(k):
        q = A @ p
        a = rr / (p @ q)
        x, r = x + a * p, r - a * q
        new = r @ r
        p, rr = r + new / rr * p, new
    return x


def _bicgstab(A, b, k):
    x, r, rh, p = np.zeros_like(b), b.copy(), b.copy(), b.copy()
    rho = rh @ r
    for _ in range(k):
        v = A @ p
        a = rho / (rh @ v)
        s = r - a * v
        t = A @ s
        w = (t @ s) / (t @ t)
        x, r = x + a * p + w * s, s - w * t
        new = rh @ r
        p, rho = r + new * a / (rho * w) * (p - w * v), new
    return x


@pytest.mark.parametrize("longest", [1, 5, 6, 7, 8])
@pytest.mark.parametrize("n", [1, 16, 17, 511, 512, 513, 1025, 8192, 8193, 148 * 512 + 1, 148 * 2 * 512,
                               148 * 2 * 512 + 33])
@pytest.mark.parametrize("empty_tile_row", [False, True])
def test_one_chunk_products_and_solves(mf, cuda, n, longest, empty_tile_row):
    import torch
    if empty_tile_row and n <= 64:
        pytest.skip("too few tile-rows to leave one empty")
    A = _banded(n, longest, seed=n + longest, empty_tile_row=empty_tile_row)
    if empty_tile_row:                                # b in the range of the singular matrix
        b = A @ np.random.default_rng(1).uniform(-1, 1, n)
    else:
        b = np.random.default_rng(2).uniform(-1, 1, n)
    G = mf.Matrix.from_csr(n, n, A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data)
    x = np.random.default_rng(3).uniform(-1, 1, n)
    ye, scale = A @ x, abs(A) @ abs(x)
    for prec, extra in (("fp64", 0.0), ("mixed", 2.0 ** -24)):
        y = G.spmv(x, precision=prec)
        assert np.all(np.abs(y - ye) <= (10 * EPS + 1.01 * extra) * scale), prec
    t = torch.from_numpy(x).cuda()
    G.spmv_noalloc(t, t, precision="fp64")            # y over x: formed from a copy
    torch.cuda.synchronize()
    np.testing.assert_array_equal(t.cpu().numpy(), G.spmv(x, precision="fp64"))
    t = torch.from_numpy(x).cuda()
    np.testing.assert_array_equal(G.spmv(t, t, precision="fp64").cpu().numpy(), G.spmv(x, precision="fp64"))
    if n < 16:
        return
    for method, plain in (("cg", _cg), ("bicgstab", _bicgstab)):
        xe = plain(A, b, 3)
        for prec, tol in (("fp64", 1e4 * EPS), ("mixed", 1e4 * 2.0 ** -24)):
            xs, rep = G.solve(b, method=method, precision=prec, max_iter=3, fixed_iters=1, replace_every=2)
            assert rep["iterations"] == 3
            assert np.linalg.norm(xs - xe) <= tol * np.linalg.norm(xe), (method, prec)
            products = 3 * (1 if method == "cg" else 2)
            if prec == "mixed":
                assert sum(rep["nnz_uses"]) == products * G.info["nnz"], (method, rep["nnz_uses"])


def test_solve_with_more_columns_than_rows_ignores_stale_memory(mf, cuda):
    """Columns past n_rows multiply zeros, whatever an earlier solve left behind."""
    n, cols = 509, 560
    A = _banded(n, 7, seed=5)
    wide = sp.csr_matrix(sp.hstack([A, sp.csr_matrix((n, cols - n))]) + sp.csr_matrix(
        (np.full(n, 0.125), (np.arange(n), n + np.arange(n) % (cols - n))), shape=(n, cols)))
    wide.sort_indices()
    G = mf.Matrix.from_csr(n, cols, wide.indptr.astype(np.int32), wide.indices.astype(np.int32), wide.data)
    b = np.random.default_rng(6).uniform(-1, 1, n)
    G.spmv(np.full(cols, np.nan))                     # nothing of this may reach the solves below
    for method, plain in (("cg", _cg), ("bicgstab", _bicgstab)):
        xe = plain(A, b, 3)
        for prec, tol in (("fp64", 1e4 * EPS), ("mixed", 1e4 * 2.0 ** -24)):
            x, _ = G.solve(b, method=method, precision=prec, max_iter=3, fixed_iters=1, replace_every=2)
            assert np.linalg.norm(x - xe) <= tol * np.linalg.norm(xe), (method, prec)
