"""Batch items solved by teams of blocks, with 1 to 8 columns, in both precisions:
a fixed number of CG iterations on every column against the same iterations in
plain FP64.  Uneven systems in one launch, so teams of several sizes and queue
items run side by side; direct launches, graph replays and initial guesses.

Bounds: these systems are diagonally dominant (condition below 100), so ten
iterations amplify rounding by less than 1e4; FP32-stored values put 2^-24 in its
place."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _cg(S, b, x0, k):
    x = x0.copy()
    r = b - S @ x
    p, rr = r.copy(), r @ r
    for _ in range(k):
        q = S @ p
        a = rr / (p @ q)
        x, r = x + a * p, r - a * q
        new = r @ r
        p, rr = r + new / rr * p, new
    return x


def _system(side, kind, rng):
    from millefeuille import matrices as M
    dirs2 = [(1, 0), (0, 1)]
    dirs3 = [(dx, dy, dz) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1) if (dz, dy, dx) > (0, 0, 0)]
    A = M._edge_stencil((side, side), dirs2, rng, 0.1) if kind == "2d" else \
        M._edge_stencil((side, side, side), dirs3, rng, 0.1)
    S = A.to_scipy().tocsr()
    S.setdiag(S.diagonal() * 1.1)
    return S


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("cap", [1, 2, 4, 8])
def test_team_items_match_plain_iterations(mf, cuda, precision, cap):
    import torch
    rng = np.random.default_rng(cap)
    specs = [("3d", 20, 2), ("2d", 100, 3), ("3d", 12, 4), ("2d", 75, 5), ("3d", 9, 1), ("2d", 60, 8), ("2d", 20, 7)]
    systems = [(_system(side, kind, rng), nr) for kind, side, nr in specs]
    mats = [mf.Matrix.from_csr(S.shape[0], S.shape[0], S.indptr.astype(np.int32), S.indices.astype(np.int32), S.data)
            for S, _ in systems]
    Bs = [rng.standard_normal((nr, S.shape[0])) for S, nr in systems]
    X0 = [rng.standard_normal(B.shape) for B in Bs]
    dB = [torch.from_numpy(B).cuda() for B in Bs]
    batch = mf.Batch(mats, [nr for _, nr in systems])
    batch.configure(cap, 1)
    tol = 1e4 * (EPS if precision == "fp64" else 2.0 ** -24)
    for guess in (0, 1):
        o = mf.default_options(precision=precision, tol=0.0, max_iter=10, fixed_iters=1, replace_every=6, x0_given=guess)
        exact = [np.stack([_cg(S, b, x if guess else 0 * x, 10) for b, x in zip(B, X)])
                 for (S, _), B, X in zip(systems, Bs, X0)]
        for graph in (False, True, True):
            dX = [torch.from_numpy(x.copy()).cuda() if guess else torch.zeros_like(b) for x, b in zip(X0, dB)]
            got, reps = batch.solve(dB, dX, options=o, use_graph=graph)
            assert max(r[0]["item_blocks"] for r in reps) > 1
            for k, (x, e) in enumerate(zip(got, exact)):
                err = np.linalg.norm(x.cpu().numpy() - e) / np.linalg.norm(e)
                assert err <= tol, (precision, cap, guess, graph, specs[k], err)
