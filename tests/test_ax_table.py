"""A x with and without the table of x (cassandra_b200/csrc/fast.cu), at the
block counts where one takes over from the other: equal to the row-major
product, exactly, on integer-valued vectors."""
import numpy as np
import pytest
import torch

import cassandra_b200 as cb
from tests.golden.make_golden import FIXTURES, SET5, SET8

pytestmark = pytest.mark.gpu

BLOCK, DIRECT = 16384, 48  # rows per block, most blocks without a table
TWELVE = SET8 + [0xC3, 0x0303, 0x81, 0x1818]  # more patterns than index words held at once, slots 8, 4, 2 and 1


@pytest.mark.parametrize("rows", [1, BLOCK - 1, BLOCK + 1, DIRECT * BLOCK, DIRECT * BLOCK + 1, 60 * BLOCK - 33])
@pytest.mark.parametrize("name,mode", [("set8", "expanded"), ("set5", "reference"), ("twelve", "reference"),
                                       ("fixtures", "reference")])
def test_products_around_the_table(cuda, rows, name, mode):
    masks = {"set8": SET8, "set5": SET5, "twelve": TWELVE, "fixtures": list(FIXTURES.values())}[name]
    g = cb.GroupIndexer(masks, mode)
    pos = cb.generate_positions(rows, rows, 10, 50)
    a = cb.MatrixCSR.from_positions(g, pos, "blocked")
    idx = g.indices(pos).long()
    x = torch.randint(-8, 9, (g.index_space_size,), device="cuda")
    want = x[idx].sum(1)
    for dt in (torch.float32, torch.float64):
        assert torch.equal((a @ x.to(dt)).long(), want)


def test_batch_crosses_the_table_bound(cuda):
    """A batch of more blocks than the direct product takes, whose problems
    retire until few are left: every problem as in its own fit."""
    sizes = [DIRECT * BLOCK // 2, 5000, 30 * BLOCK + 7]
    g = cb.GroupIndexer(SET5[3:], "reference")
    n = sum(sizes)
    pos = cb.generate_positions(3, n, 20, 40)
    b = torch.from_numpy(np.random.RandomState(0).randint(-20, 21, n)).double().cuda()
    xs, reps, ok = cb.solve_batched(cb.MatrixCSR.from_positions_batched(g, pos, sizes), b, precision="fp64", tol=1e-10)
    assert ok
    row = 0
    for q, m in enumerate(sizes):
        s = cb.PCG(cb.MatrixCSR.from_positions(g, pos[row:row + m].contiguous(), "blocked"), b[row:row + m].contiguous(),
                   tol=1e-10, max_iterations=20000)
        assert s.run()["converged"]
        assert float((xs[q] - s.x()).norm() / s.x().norm()) < 1e-6  # two solves to 1e-10 of the same system
        row += m
