"""The operand of a product is read where it is only when a kernel can read it there;
what a copy of it takes, the product takes, and what a copy refuses, it refuses."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def case(mf, cuda):
    import torch
    from millefeuille import matrices as M
    A = M.laplace2d(37)
    G = mf.Matrix.from_csr(A.n, A.n, A.rowptr, A.colidx, A.val)
    x = np.random.default_rng(1).standard_normal(A.n)
    y = torch.zeros(A.n, dtype=torch.float64, device=cuda)
    return G, x, y, G.spmv(x)


def _calls(G, mf):
    from millefeuille import _lib
    L = _lib.load()
    return {"mf_spmv": lambda x, y: L.mf_spmv(G._h, C.c_void_p(x), C.c_void_p(y), mf.MF_PREC_FP64, 1, None, None),
            "mf_spmv_noalloc": lambda x, y: L.mf_spmv_noalloc(G._h, C.c_void_p(x), C.c_void_p(y), mf.MF_PREC_FP64, None)}


@pytest.mark.parametrize("entry", ["mf_spmv", "mf_spmv_noalloc"])
@pytest.mark.parametrize("offset", [1, 4, 8])
def test_operand_on_any_byte_boundary(mf, case, entry, offset):
    import torch
    G, x, y, want = case
    raw = torch.zeros(8 * x.size + 16, dtype=torch.uint8, device=y.device)
    raw[offset:offset + 8 * x.size] = torch.from_numpy(x.view(np.uint8)).to(y.device)
    torch.cuda.synchronize()
    assert _calls(G, mf)[entry](raw.data_ptr() + offset, y.data_ptr()) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(y.cpu().numpy(), want)


@pytest.mark.parametrize("entry", ["mf_spmv", "mf_spmv_noalloc"])
def test_pageable_host_operand_is_refused(mf, case, entry):
    import torch
    from millefeuille import _lib
    G, x, y, want = case
    assert _calls(G, mf)[entry](x.ctypes.data, y.data_ptr()) == _lib.MF_ERR_CUDA
    t = torch.from_numpy(x).to(y.device)                 # and the device still works
    torch.cuda.synchronize()
    assert _calls(G, mf)[entry](t.data_ptr(), y.data_ptr()) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(y.cpu().numpy(), want)
