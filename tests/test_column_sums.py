"""Column sums of A'y's partials (cassandra_b200/csrc/fast.cuh, fast_col_sum):
batches of 32 and 16 and their remainders by halves.  A forced schedule gives a
column as many partials as the layout has blocks; exact on integer-valued
vectors, and through the solvers' steps against the residual in 64 bits."""
import numpy as np
import pytest
import torch

import cassandra_b200 as cb

pytestmark = pytest.mark.gpu

BLOCK = 16384


@pytest.mark.parametrize("blocks", [1, 2, 3, 5, 7, 8, 15, 16, 17, 31, 32, 33, 47, 63])
def test_partials_of_every_number(cuda, monkeypatch, blocks):
    monkeypatch.setenv("CAS_ATY_SCHEDULE", "4,0,16,0,1")  # an item per block: 2,368 items wanted
    g = cb.GroupIndexer([0xFF], "reference")  # 3321 columns, one super-chunk
    rows = blocks * BLOCK - 3
    pos = cb.generate_positions(blocks, rows, 10, 50)
    a = cb.MatrixCSR.from_positions(g, pos, "blocked")
    y = torch.randint(-2, 3, (rows,), device="cuda")
    idx = g.indices(pos).long()
    want = torch.zeros(g.index_space_size, dtype=torch.long, device="cuda")
    want.index_add_(0, idx.flatten(), y.repeat_interleave(idx.shape[1]))
    for dt in (torch.float32, torch.float64):
        assert torch.equal(a.rmatvec(y.to(dt)).long(), want)


@pytest.mark.parametrize("blocks", [5, 17, 47])
@pytest.mark.parametrize("solver", [cb.PCG, cb.LSQR, cb.LSMR])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_steps_of_the_solvers(cuda, monkeypatch, blocks, solver, precision):
    monkeypatch.setenv("CAS_ATY_SCHEDULE", "4,0,16,0,1")
    g = cb.GroupIndexer([0xFF], "reference")
    rows = blocks * BLOCK - 3
    pos = cb.generate_positions(blocks, rows, 20, 40)
    b = torch.from_numpy(np.random.RandomState(blocks).randint(-20, 21, rows)).double().cuda()
    s = solver(cb.MatrixCSR.from_positions(g, pos, "blocked"), b, precision=precision, tol=1e-8)
    assert s.run()["converged"]
    idx = g.indices(pos).long()
    res = []
    for v in (b - s.x()[idx].sum(1), b):
        t = torch.zeros(g.index_space_size, dtype=torch.float64, device="cuda")
        res.append(float(t.index_add_(0, idx.flatten(), v.repeat_interleave(idx.shape[1])).norm()))
    # the solver's own FP64 residual met 1e-8; this one differs by the rounding
    # of the products, far below a hundredth of it
    assert res[0] <= 1.01e-8 * res[1]
