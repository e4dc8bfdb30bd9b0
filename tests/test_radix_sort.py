"""The transposed copy's radix sort (cassandra_b200/csrc/csr.cu): column
counts around each number of 9-bit passes, entry counts around its tiles of
8,192, and columns that crowd: the rows of every column in order and diag(A'A), exactly."""
import numpy as np
import pytest
import torch

import cassandra_b200 as cb

pytestmark = pytest.mark.gpu

TILE = 8192


@pytest.mark.parametrize("cols", [1, 2, 512, 513, 1 << 17, 1 << 18, (1 << 18) + 1, (1 << 22) + 3])
@pytest.mark.parametrize("rows,k", [(1, 1), (TILE - 1, 1), (TILE, 1), (TILE + 1, 1), (1171, 7), (3 * TILE + 5, 2),
                                    (5000, 34)])
@pytest.mark.parametrize("kind", ["even", "crowded"])
def test_rows_of_every_column_in_order(cuda, cols, rows, k, kind):
    rng = np.random.RandomState(rows + cols % 1000)
    idx = rng.randint(0, cols, (rows, k))
    if kind == "crowded":  # most entries in the last column and a run of equal low digits
        idx = np.where(rng.rand(rows, k) < 0.7, cols - 1, idx - idx % 512)
    a = cb.MatrixCSR.from_indices(torch.from_numpy(idx.astype(np.int32)).cuda(), cols)
    col_ptr, row_idx = a.transposed()
    flat = idx.reshape(-1)
    order = np.argsort(flat, kind="stable")
    assert np.array_equal(row_idx.cpu().numpy().astype(np.int64), order // k)
    assert np.array_equal(col_ptr.cpu().numpy(), np.searchsorted(flat[order], np.arange(cols + 1)))
    # diag(A'A): the squares of a column's copies in each row
    pair, copies = np.unique(np.arange(rows).repeat(k) * np.int64(cols) + flat, return_counts=True)
    diag = np.bincount(pair % cols, copies.astype(np.float64) ** 2, cols)
    with np.errstate(divide="ignore"):
        want = 1.0 / diag  # empty columns: inf
    assert np.array_equal(cb.jacobi_preconditioner_of_ata(a).cpu().numpy(), want)
