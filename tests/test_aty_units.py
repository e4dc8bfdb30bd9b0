"""The work units of A'y (cassandra_b200/csrc/fast.cu): items split by columns
where the entries of their first block pass equal shares.  Exact on
integer-valued vectors, from one row to more items than are split, with the
entries spread by play or crowded into a few columns, at aligned and
unaligned y; and in a batch whose units are laid out again as problems
retire."""
import numpy as np
import pytest
import torch

import cassandra_b200 as cb
from tests.golden.make_golden import FIXTURES, SET5, SET8

pytestmark = pytest.mark.gpu

BLOCK = 16384


def _positions(kind, rows):
    if kind == "play":
        return cb.generate_positions(rows, rows, 10, 50)
    few = cb.generate_positions(7, {"one": 1, "three": 3}[kind], 10, 50)
    return few[torch.arange(rows, device="cuda") * len(few) // rows].contiguous()


@pytest.mark.parametrize("rows", [1, 33, BLOCK - 1, 2 * BLOCK + 1, 9 * BLOCK, 40 * BLOCK - 5])
@pytest.mark.parametrize("kind", ["play", "one", "three"])
@pytest.mark.parametrize("name,mode", [("set8", "expanded"), ("set5", "reference"), ("fixtures", "reference")])
def test_split_items_cover_every_column(cuda, rows, kind, name, mode):
    g = cb.GroupIndexer({"set8": SET8, "set5": SET5, "fixtures": list(FIXTURES.values())}[name], mode)
    pos = _positions(kind, rows)
    a = cb.MatrixCSR.from_positions(g, pos, "blocked")
    idx = g.indices(pos).long()
    # |sum| < 2^24 in every column: at most 8 copies of a column a row
    top = 3 if rows * 8 * 3 < 2**24 else 1
    y = torch.randint(-top, top + 1, (rows + 1,), device="cuda")
    for shift in (0, 1):
        v = y[shift:shift + rows]
        want = torch.zeros(g.index_space_size, dtype=torch.long, device="cuda")
        want.index_add_(0, idx.flatten(), v.repeat_interleave(idx.shape[1]))
        for dt in (torch.float32, torch.float64):
            w = torch.empty(rows + 1, device="cuda", dtype=dt)[shift:shift + rows].copy_(v)
            assert torch.equal(a.rmatvec(w).long(), want)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_batch_lays_units_out_again(cuda, precision):
    """Problems of several sizes that retire one by one: the residual of each
    in 64 bits, from the index table."""
    sizes = [9 * BLOCK, 7 * BLOCK + 1, 5000, 17 * BLOCK - 3, 1]
    g = cb.GroupIndexer(SET5[3:], "reference")
    n = sum(sizes)
    pos = cb.generate_positions(3, n, 20, 40)
    b = torch.from_numpy(np.random.RandomState(0).randint(-20, 21, n)).double().cuda()
    tol = 1e-8
    xs, reps, ok = cb.solve_batched(cb.MatrixCSR.from_positions_batched(g, pos, sizes), b, precision=precision, tol=tol)
    assert ok
    idx = g.indices(pos).long()
    row = 0
    for q, m in enumerate(sizes):
        i, bq = idx[row:row + m], b[row:row + m]
        res = []
        for v in (bq - xs[q].double()[i].sum(1), bq):
            t = torch.zeros(g.index_space_size, dtype=torch.float64, device="cuda")
            res.append(float(t.index_add_(0, i.flatten(), v.repeat_interleave(i.shape[1])).norm()))
        # the solver's own FP64 residual met tol; ours differs by the rounding
        # of the products, 1e-16 * sqrt(entries) of |A'b|-sized terms: far below
        # a hundredth of tol
        assert res[0] <= 1.01 * tol * res[1]
        row += m
