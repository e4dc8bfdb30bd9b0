"""A x on the rows layout (cassandra_b200/csrc/csr.cu): a warp takes four rows
at a time; row counts around that and entries a row around a warp, exact on
integer-valued vectors."""
import pytest
import torch

import cassandra_b200 as cb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 31, 1001, 100_003])
@pytest.mark.parametrize("k", [1, 7, 32, 33, 64])
def test_rows_in_fours(cuda, rows, k):
    cols = 1 + rows // 3
    g = torch.Generator(device="cuda").manual_seed(rows + k)
    idx = torch.randint(cols, (rows, k), generator=g, device="cuda", dtype=torch.int32)
    x = torch.randint(-8, 9, (cols,), generator=g, device="cuda")
    a = cb.MatrixCSR.from_indices(idx, cols)
    for dt in (torch.float32, torch.float64):
        assert torch.equal((a @ x.to(dt)).long(), x[idx.long()].sum(1))
