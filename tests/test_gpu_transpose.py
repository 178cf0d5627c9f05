"""Transposed handles, exactly: every array of the handle for A^T against the
oracle's tiles of the transpose (SciPy's CSC arrays: each row of A^T keeps the
order of A's rows).  The sizes are the edges of the sort on the device: digits
(256 and 65,536 columns) and blocks (4,096 entries), empty columns, one very
long column, and matrices whose first row pointer is not zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ["tile_ptr", "tile_columnidx", "csr_offset", "csrptr_offset", "val", "val_low", "col", "ptr",
        "nonzero_row_new", "blockrowid_new", "blockcsr_ptr_new", "tile_rowidx", "block_signal"]


def _entries(n_rows, n_cols, nnz, seed, long_column=False):
    """nnz distinct positions, row by row with unsorted columns, as (rowptr, colidx, val)."""
    rng = np.random.default_rng(seed)
    at = np.sort(rng.choice(n_rows * n_cols, size=nnz, replace=False))
    rows, cols = at // n_cols, at % n_cols
    if long_column:
        rest = cols != n_cols // 2
        rows = np.concatenate([rows[rest], np.arange(n_rows)])
        cols = np.concatenate([cols[rest], np.full(n_rows, n_cols // 2)])
    order = np.lexsort((rng.random(rows.size), rows))
    rows, cols = rows[order], cols[order]
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n_rows))]).astype(np.int32)
    return rowptr, cols.astype(np.int32), rng.standard_normal(rows.size)


def _check(mf, oracle_mod, T, n_rows, n_cols, rowptr, colidx, val, low=None):
    """T against the transpose of the rows' entries from rowptr[0] on."""
    rows = np.repeat(np.arange(n_rows), np.diff(rowptr))
    lo, hi = int(rowptr[0]), int(rowptr[-1])
    order = np.argsort(colidx[lo:hi], kind="stable")
    tptr = np.concatenate([[0], np.cumsum(np.bincount(colidx[lo:hi], minlength=n_cols))]).astype(np.int32)
    want = oracle_mod.Tiles(n_cols, n_rows, tptr, rows[order].astype(np.int32), val[lo:hi][order]).arrays()
    if low is not None:
        want["val_low"] = oracle_mod.Tiles(n_cols, n_rows, tptr, rows[order].astype(np.int32),
                                           low[lo:hi][order].astype(np.float64)).arrays()["val_low"]
    assert T.info["n_rows"] == n_cols and T.info["n_cols"] == n_rows and T.info["nnz"] == hi - lo
    for k in KEYS:
        np.testing.assert_array_equal(T.export(k), want[k], err_msg=k)


@pytest.mark.parametrize("n_rows,n_cols,nnz,long_column", [
    (40, 30, 0, False), (1, 1, 1, False), (40, 30, 1, False),
    (300, 255, 4095, False), (300, 256, 4096, False), (300, 257, 4097, False),
    (17, 65536, 9000, False), (33, 65537, 12289, False), (500, 70000, 20000, False),
    (70001, 300, 70001, True), (9000, 2000, 30000, False),
])
def test_transposed_handle_is_exact(mf, oracle_mod, cuda, n_rows, n_cols, nnz, long_column):
    rowptr, colidx, val = _entries(n_rows, n_cols, nnz, n_cols, long_column)
    G = mf.Matrix.from_csr(n_rows, n_cols, rowptr, colidx, val)
    _check(mf, oracle_mod, G.transposed(), n_rows, n_cols, rowptr, colidx, val)


def test_transposed_handle_with_low_values_and_shifted_rows(mf, oracle_mod, cuda):
    """Separate FP32 values travel with their entries; entries before the first row
    pointer stay out."""
    rowptr, colidx, val = _entries(400, 600, 9000, 3)
    low = (val * 1.5).astype(np.float32)
    first = 37
    G = mf.Matrix.from_csr(400 - first, 600, rowptr[first:], colidx, val, val_low=low)
    assert rowptr[first] > 0
    _check(mf, oracle_mod, G.transposed(), 400 - first, 600, rowptr[first:], colidx, val, low)


def test_transposing_twice_gives_the_matrix_back(mf, oracle_mod, cuda):
    rowptr, colidx, val = _entries(1000, 700, 20000, 5)
    for r in range(1000):                       # sorted rows: the transpose's transpose has them sorted
        s = slice(rowptr[r], rowptr[r + 1])
        o = np.argsort(colidx[s])
        colidx[s], val[s] = colidx[s][o], val[s][o]
    G = mf.Matrix.from_csr(1000, 700, rowptr, colidx, val)
    B = G.transposed().transposed()
    for k in KEYS:
        np.testing.assert_array_equal(B.export(k), G.export(k), err_msg=k)
