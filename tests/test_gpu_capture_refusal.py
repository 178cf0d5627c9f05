"""Calls that allocate, on a stream that is being captured, are refused as they always
were (they synchronise), and leave the handle as it was: the same calls work after
the capture."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [1, 2], ids=["thread_local", "relaxed"])
@pytest.mark.parametrize("warm", [False, True])
def test_refused_under_capture_and_sound_after(mf, cuda, mode, warm):
    import torch
    from millefeuille import _lib
    from millefeuille import matrices as M
    L = _lib.load()
    rt = C.CDLL("libcudart.so.12")
    A = M.laplace2d(50)
    S = A.to_scipy().tocsr()
    G = mf.Matrix.from_csr(A.n, A.n, A.rowptr, A.colidx, A.val)
    b = np.random.default_rng(0).standard_normal((4, A.n))
    B = torch.from_numpy(b).to(cuda)
    X = torch.zeros_like(B)
    if warm:
        G.solve(B[0].contiguous(), precision="fp64", tol=1e-10)
    o = mf.default_options(precision="fp64", tol=1e-10)
    torch.cuda.synchronize()
    stream, graph, h = C.c_void_p(), C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamCreateWithFlags(C.byref(stream), 1) == 0
    calls = {
        "multi": lambda s: L.mf_solve_multi(G._h, 4, C.c_void_p(B.data_ptr()), C.c_void_p(X.data_ptr()), C.byref(o),
                                            None, 1, s),
        "host": lambda s: L.mf_solve(G._h, b.ctypes.data_as(C.c_void_p), b.copy().ctypes.data_as(C.c_void_p),
                                     C.byref(o), None, 0, s),
        "transposed": lambda s: L.mf_matrix_create_transposed(C.byref(h), G._h, s),
    }
    for name, call in calls.items():
        assert rt.cudaStreamBeginCapture(stream, mode) == 0
        assert call(stream) == _lib.MF_ERR_CUDA, name
        rt.cudaStreamEndCapture(stream, C.byref(graph))
        rt.cudaGetLastError()
    x, _ = G.solve_multi(B, precision="fp64", tol=1e-10, stream=stream.value)
    assert np.abs((S @ x.cpu().numpy().T).T - b).max() < 1e-6
    x, _ = G.solve(b[1], precision="fp64", tol=1e-10, stream=stream.value)
    assert np.abs(S @ x - b[1]).max() < 1e-6
    T = G.transposed(stream=stream.value)
    assert np.abs(T.spmv(b[2], stream=stream.value) - S.T @ b[2]).max() < 1e-10
    T.close()
    assert rt.cudaStreamDestroy(stream) == 0
