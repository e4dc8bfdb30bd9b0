"""Which slices of x the table A x stages (cassandra_b200/csrc/fast.cu,
table_plan): one pattern whose slice fits but pays only from some 270 blocks
on, and a set whose patterns join one by one; exact on integer-valued
vectors, in a batch too."""
import pytest
import torch

import cassandra_b200 as cb
from tests.golden.make_golden import SET5

pytestmark = pytest.mark.gpu

BLOCK = 16384


@pytest.mark.parametrize("blocks", [49, 122, 300])
@pytest.mark.parametrize("masks", [SET5[:1], SET5])
def test_slices_that_pay(cuda, blocks, masks):
    rows = blocks * BLOCK - 7
    g = cb.GroupIndexer(masks, "reference")
    pos = cb.generate_positions(blocks, rows, 10, 50)
    a = cb.MatrixCSR.from_positions(g, pos, "blocked")
    idx = g.indices(pos)
    x = torch.randint(-8, 9, (g.index_space_size,), device="cuda")
    want = sum(x[idx[:, s].long()] for s in range(idx.shape[1]))
    for dt in (torch.float32, torch.float64):
        assert torch.equal((a @ x.to(dt)).long(), want)


def test_batch(cuda):
    sizes = [30 * BLOCK + 1, 5, 0, 40 * BLOCK]
    g = cb.GroupIndexer(SET5, "reference")
    pos = cb.generate_positions(8, sum(sizes), 10, 50)
    a = cb.MatrixCSR.from_positions_batched(g, pos, sizes)
    cols = g.index_space_size
    q = torch.arange(len(sizes), device="cuda").repeat_interleave(torch.tensor(sizes, device="cuda"))
    x = torch.randint(-8, 9, (cols * len(sizes),), device="cuda")
    want = x[g.indices(pos).long() + (q * cols)[:, None]].sum(1)
    for dt in (torch.float32, torch.float64):
        assert torch.equal((a @ x.to(dt)).long(), want)
