"""A stream that one thread is capturing survives what another thread does with its
own handles and its own stream: making, solving, growing workspaces, destroying.
(Captures in thread-local mode on a non-blocking and on a blocking stream; device-wide
synchronisation and the legacy stream would end them with an error.)"""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THREAD_LOCAL = 1


def _use_handles(mf, stream):
    """Everything that allocates or frees, on `stream`; returns the largest error of its solves."""
    from millefeuille import matrices as M
    worst = 0.0
    for side in (12, 70):
        A = M.laplace2d(side)
        S = A.to_scipy().tocsr()
        b = np.ones(A.n)
        G = mf.Matrix.from_csr(A.n, A.n, A.rowptr, A.colidx, A.val, stream=stream)
        for bps in (0, 1):                                        # a second workspace replaces the first
            x, _ = G.solve(b, precision="fp64", tol=1e-10, stream=stream, blocks_per_sm=bps)
            worst = max(worst, float(np.abs(S @ x - b).max()))
        for nrhs in (2, 9):                                       # wider columns, more result slots
            B = np.ones((nrhs, A.n))
            X, _ = G.solve_multi(B, precision="fp64", tol=1e-10, stream=stream)
            worst = max(worst, float(np.abs((S @ X.T).T - B).max()))
        y = G.spmv(b, stream=stream)                              # host arrays: the staging grows with the call
        worst = max(worst, float(np.abs(y - S @ b).max()))
        T = G.transposed(stream=stream)
        T.close()
        G.close()
    return worst


@pytest.mark.parametrize("flags", [1, 0], ids=["non_blocking", "blocking"])
def test_capture_in_another_thread_survives(mf, cuda, flags):
    import torch
    torch.zeros(1, device=cuda)
    rt = C.CDLL("libcudart.so.12")
    captured, own, graph = C.c_void_p(), C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamCreateWithFlags(C.byref(captured), flags) == 0
    assert rt.cudaStreamCreateWithFlags(C.byref(own), 1) == 0
    _use_handles(mf, own.value)                                   # first use of everything outside the capture
    result = []
    assert rt.cudaStreamBeginCapture(captured, THREAD_LOCAL) == 0

    def work():
        try:
            torch.cuda.set_device(0)
            result.append(_use_handles(mf, own.value))
        except Exception as e:                                    # reported below, after the capture has ended
            result.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    ended = rt.cudaStreamEndCapture(captured, C.byref(graph))
    rt.cudaGetLastError()
    assert isinstance(result[0], float), result[0]
    assert result[0] < 1e-6
    assert ended == 0
    assert rt.cudaGraphDestroy(graph) == 0
    assert rt.cudaStreamDestroy(captured) == 0 and rt.cudaStreamDestroy(own) == 0
