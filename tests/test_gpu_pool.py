"""The library's memory pool keeps at most 1 GiB beyond what is live: a destroyed
handle's memory is there for others at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GIB = 1 << 30


def _tridiagonal(n, cuda):
    """rowptr, colidx, val of a tridiagonal matrix, on the device."""
    import torch
    i = torch.arange(n, device=cuda, dtype=torch.int32)
    cols = torch.stack([i - 1, i, i + 1], dim=1).reshape(-1)[1:-1].contiguous()
    rowptr = torch.clamp(3 * torch.arange(n + 1, device=cuda, dtype=torch.int32) - 1, 0, 3 * n - 2)
    return rowptr, cols, torch.ones(3 * n - 2, dtype=torch.float64, device=cuda)


def test_destroyed_handles_give_their_memory_back(mf, cuda):
    import torch
    n = 12_000_000
    csr = _tridiagonal(n, cuda)
    torch.cuda.synchronize()
    small = mf.Matrix.from_csr(1000, 1000, *_tridiagonal(1000, cuda))
    free0 = torch.cuda.mem_get_info()[0]
    for keep in (True, False):                      # beside a live handle, and with nothing live
        if not keep:
            small.close()
        G = mf.Matrix.from_csr(n, n, *csr)
        assert free0 - torch.cuda.mem_get_info()[0] > 2 * GIB
        G.close()
        assert free0 - torch.cuda.mem_get_info()[0] < 1.1 * GIB
