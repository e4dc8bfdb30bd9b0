"""A x on the rows layout (cassandra_b200/csrc/csr.cu): rows of up to 64
entries go four to a warp, longer ones one; entries a row around that, exact
on integer-valued vectors."""
import pytest
import torch

import cassandra_b200 as cb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 5, 9, 1001, 20_003])
@pytest.mark.parametrize("k", [63, 64, 65, 96, 129, 1000])
def test_rows_around_the_bound(cuda, rows, k):
    cols = 1 + rows // 3
    g = torch.Generator(device="cuda").manual_seed(rows + k)
    idx = torch.randint(cols, (rows, k), generator=g, device="cuda", dtype=torch.int32)
    x = torch.randint(-8, 9, (cols,), generator=g, device="cuda")
    a = cb.MatrixCSR.from_indices(idx, cols)
    for dt in (torch.float32, torch.float64):
        assert torch.equal((a @ x.to(dt)).long(), x[idx.long()].sum(1))
