"""Batched solves of one problem: the active list takes the units that the
layout was built with (cassandra_b200/csrc/fast.cuh, fast_plan_active).  One
and several super-chunks, items range by range and not, the default schedule,
a forced and a tuned one, every entry point that leads there; the residual in
64 bits from the index table."""
import numpy as np
import pytest
import torch

import cassandra_b200 as cb
from tests.golden.make_golden import SET5, SET8

pytestmark = pytest.mark.gpu

BLOCK = 16384
TOL = 1e-8
MOST = 60000  # the system of 49,153 rows and 166,212 columns takes 18,600 (FP64) to 21,400 (mixed) iterations
SETS = {"set8": SET8, "set5": SET5, "narrow": [0xFF]}  # narrow: 3321 columns, one super-chunk


def _residual(idx, cols, b, x):
    """||A'(b - A x)|| / ||A'b||."""
    norm = []
    for v in (b - x[idx].sum(1), b):
        t = torch.zeros(cols, dtype=torch.float64, device="cuda")
        norm.append(float(t.index_add_(0, idx.flatten(), v.repeat_interleave(idx.shape[1])).norm()))
    return norm[0] / norm[1]


def _solve(entry, g, pos, b, precision):
    n = len(pos)
    if entry == "fit":
        return cb.fit_weights_batched(g, pos, b, [n], precision=precision, tol=TOL, max_iterations=MOST)
    a = cb.MatrixCSR.from_positions_batched(g, pos, [n]) if entry == "batched" else \
        cb.MatrixCSR.from_positions(g, pos, "blocked")
    return cb.solve_batched(a, b, precision=precision, tol=TOL, max_iterations=MOST)


def _check(name, mode, rows, entry, precision):
    g = cb.GroupIndexer(SETS[name], mode)
    pos = cb.generate_positions(rows, rows, 20, 40)
    b = torch.from_numpy(np.random.RandomState(rows).randint(-20, 21, rows)).double().cuda()
    x, reps, ok = _solve(entry, g, pos, b, precision)
    assert ok and x.shape == (1, g.index_space_size) and len(reps) == 1
    assert reps[0]["converged"] and 0 < reps[0]["iterations"] < MOST
    # the solver's own FP64 residual met TOL; this one differs by the rounding
    # of the products, far below a hundredth of TOL
    assert _residual(g.indices(pos).long(), g.index_space_size, b, x[0]) <= 1.01 * TOL


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("entry", ["batched", "plain", "fit"])
@pytest.mark.parametrize("name,mode", [("set8", "expanded"), ("set5", "reference"), ("narrow", "reference")])
@pytest.mark.parametrize("rows", [1, 5000, 3 * BLOCK + 1])
def test_one_problem(cuda, rows, name, mode, entry, precision):
    _check(name, mode, rows, entry, precision)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("schedule", ["4,0,2,0,0", "4,1,4,0,1", "2,1,4,1,1"])
def test_forced_schedules(cuda, monkeypatch, schedule, precision):
    monkeypatch.setenv("CAS_ATY_SCHEDULE", schedule)
    _check("set5", "reference", 4 * BLOCK - 3, "batched", precision)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_tuned_schedule(cuda, precision):
    """64 blocks and more: the FP32 schedule is the autotuner's choice."""
    _check("set5", "reference", 65 * BLOCK + 5, "plain", precision)


def test_zero_targets_retire_at_setup(cuda):
    g = cb.GroupIndexer(SET8, "expanded")
    a = cb.MatrixCSR.from_positions_batched(g, cb.generate_positions(5, 4000, 20, 40), [4000])
    for precision in ("mixed", "fp64"):
        x, reps, ok = cb.solve_batched(a, torch.zeros(4000, dtype=torch.float64, device="cuda"), precision=precision)
        assert ok and reps[0]["iterations"] == 0 and torch.count_nonzero(x) == 0
