"""A cudaDeviceReset takes the process's device memory along.  Handles made after it
work, and destroying those from before it touches nothing of theirs (a fresh
context hands out the same addresses again)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import ctypes as C
import numpy as np
import millefeuille as mf
from millefeuille import matrices as M

A = M.laplace2d(60)
S = A.to_scipy().tocsr()
b = np.random.default_rng(0).standard_normal(A.n)
rt = C.CDLL("libcudart.so.12")


def handle():
    return mf.Matrix.from_csr(A.n, A.n, A.rowptr, A.colidx, A.val)


def check(G):
    x, _ = G.solve(b, precision="fp64", tol=1e-10)
    assert np.linalg.norm(S @ x - b) <= 1e-9 * np.linalg.norm(b)
    X, _ = G.solve_multi(np.stack([b, 2 * b]), precision="fp64", tol=1e-10)
    assert np.linalg.norm(S @ X[1] - 2 * b) <= 2e-9 * np.linalg.norm(b)
    T = G.transposed()
    y = T.spmv(b)
    T.close()
    assert np.abs(y - S.T @ b).max() <= 1e-12 * np.abs(b).max()


for _ in range(2):
    before = [handle(), handle()]
    for G in before:
        check(G)
    batch = mf.Batch(before, [1, 2])
    assert rt.cudaDeviceReset() == 0
    after = handle()
    check(after)
    batch.close()
    for G in before:
        G.close()
    check(after)
    kept = handle()          # would take over what the old handles' frees had given away
    check(kept)
    check(after)
    after.close()
    kept.close()
print("reset ok")
"""


def test_handles_after_a_device_reset(mf, cuda):
    env = dict(os.environ)
    env["PYTHONPATH"] = os.pathsep.join([os.path.join(ROOT, "mille-feuille_b200"), env.get("PYTHONPATH", "")])
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "reset ok" in r.stdout, r.stdout + r.stderr
