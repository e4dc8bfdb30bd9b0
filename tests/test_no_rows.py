"""Solves on a blocked layout without rows: the column sums find the tables of
empty work lists, and zeros are the solution."""
import numpy as np
import pytest
import torch

import cassandra_b200 as cb
from tests.golden.make_golden import SET8

pytestmark = pytest.mark.gpu


def _nothing():
    return (torch.empty((0, 2), dtype=torch.int64, device="cuda"), torch.empty(0, dtype=torch.float64, device="cuda"))


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("sizes", [[0], [0, 0, 0]])
def test_batched(cuda, sizes, precision):
    pos, b = _nothing()
    g = cb.GroupIndexer(SET8, "expanded")
    x, reps, ok = cb.solve_batched(cb.MatrixCSR.from_positions_batched(g, pos, sizes), b, precision=precision)
    assert ok and x.shape == (len(sizes), g.index_space_size) and not torch.count_nonzero(x)
    assert all(r["iterations"] == 0 for r in reps)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("layout", ["rows", "blocked"])
def test_single(cuda, layout, precision):
    pos, b = _nothing()
    a = cb.MatrixCSR.from_positions(cb.GroupIndexer(SET8, "reference"), pos, layout)
    assert not torch.count_nonzero(a.rmatvec(b)) and (a @ torch.ones(a.cols(), device="cuda")).numel() == 0
    if layout == "blocked" or precision == "fp64":
        s = cb.PCG(a, b, precision=precision, tol=1e-8)
        assert s.run()["converged"] and not torch.count_nonzero(s.x())


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_fit_weights(cuda, precision):
    w, rep = cb.fit_weights(SET8, np.empty((0, 2), np.uint64), np.empty(0, np.float32), precision=precision)
    assert rep["converged"] and not np.any(w)
