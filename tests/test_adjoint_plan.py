"""The adjoint's units (cassandra_b200/csrc/fast.cu, plan_splits): block counts
whose items are a part of a wave, just fill it and need more than one; the
gradient exact on integer-valued vectors, on ranges that start anywhere."""
import ctypes as C

import pytest
import torch

import cassandra_b200 as cb
from cassandra_b200 import _lib as L
from tests.golden.make_golden import SET5, SET8

pytestmark = pytest.mark.gpu

BLOCK = 16384


@pytest.mark.parametrize("name,mode", [("set8", "expanded"), ("set8", "reference"), ("set5", "reference"),
                                       ("narrow", "reference")])
def test_gradient_around_a_wave(cuda, name, mode):
    g = cb.GroupIndexer({"set8": SET8, "set5": SET5, "narrow": [0xFF]}[name], mode)
    blocks = 33
    rows = blocks * BLOCK - 5
    pos = cb.generate_positions(4, rows, 10, 50)
    a = cb.MatrixCSR.from_positions(g, pos, "blocked")
    y = torch.randint(-2, 3, (rows,), device="cuda")
    idx = g.indices(pos).long()
    for b0, b1 in [(0, 1), (0, 4), (2, 8), (1, 9), (0, 10), (5, 21), (9, blocks), (0, blocks), (blocks - 1, blocks)]:
        r0, r1 = b0 * BLOCK, min(b1 * BLOCK, rows)
        want = torch.zeros(g.index_space_size, dtype=torch.long, device="cuda")
        want.index_add_(0, idx[r0:r1].flatten(), y[r0:r1].repeat_interleave(idx.shape[1]))
        v = y[r0:r1].float()
        got = torch.empty(g.index_space_size, device="cuda")
        L.check(L.load().cas_eval_backward(a.handle, r0, r1, C.c_void_p(v.data_ptr()), C.c_void_p(got.data_ptr()),
                                           C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        assert torch.equal(got.long(), want)
