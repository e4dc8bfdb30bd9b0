"""A'y and A x of more than 2^31 rows of one entry each (a fully symmetric
pattern; the layout takes up to 2^32 entries): exact, at rows on both sides of
2^31 and at the last, unfilled block."""
import pytest
import torch

import cassandra_b200 as cb
from cassandra_b200 import _lib as L

pytestmark = pytest.mark.gpu

CORNERS = 0x8100000000000081  # one entry a row
ROWS = 2**31 + 3 * 16384 + 5
AT = [0, 1, 16383, 16384, 5 * 16384 + 7, 2**30 + 1, 2**31 - 1, 2**31, 2**31 + 1, ROWS - 6, ROWS - 1]


def test_rows_past_2_to_the_31(cuda):
    L.load().cas_release_cached_memory()
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 120 << 30:
        pytest.skip("needs 120 GB of free device memory")
    g = cb.GroupIndexer([CORNERS], "reference")
    assert g.nnz_per_row == 1
    at = torch.tensor(AT, device="cuda")
    pos = torch.zeros((ROWS, 2), dtype=torch.int64, device="cuda")
    pos[at] = cb.generate_positions(9, len(AT), 4, 10)
    cols = g.indices(pos[at].contiguous()).flatten().long()
    empty = int(g.indices(pos[2:3].contiguous())[0, 0])
    a = cb.MatrixCSR.from_positions(g, pos, "blocked")
    del pos
    value = torch.arange(1, len(AT) + 1, device="cuda")
    for dt in (torch.float32, torch.float64):
        y = torch.zeros(ROWS, dtype=dt, device="cuda")
        y[at] = value.to(dt)
        y[100] = 1000
        want = torch.zeros(g.index_space_size, dtype=dt, device="cuda")
        want.index_add_(0, cols, value.to(dt))
        want[empty] += 1000
        assert torch.equal(a.rmatvec(y), want)
        del y
        x = torch.arange(2, g.index_space_size + 2, device="cuda", dtype=dt)
        ax = a @ x
        assert torch.equal(ax[at], x[cols]) and int((ax != x[empty]).sum()) == int((cols != empty).sum())
        del ax
    del a
    L.load().cas_release_cached_memory()
    torch.cuda.empty_cache()
