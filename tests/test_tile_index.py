"""The matrix form of the indexers (cassandra_b200/csrc/tile_index.cuh): a CPU
model of the fragment order, and the kernels at the edges of their tiles
against the oracle."""
import ctypes as C

import numpy as np
import pytest
import torch

import cassandra_b200 as cb
from cassandra_b200 import _lib as L
from tests.golden.make_golden import FIXTURES, SET5, SET8

LONG = [0x0F0F0F, 0x3FFF]  # 12 and 14 squares: the general kernel
MANY = [int(m) for m in np.random.RandomState(3).choice(np.arange(1, 2048), 40, replace=False)]  # 40 tiles: two chunks


def _square(t, s, b, r):
    """The square of byte b of register r of k-step s, lane t of a quad."""
    return 2 * t + s + 8 * b + 32 * r


def test_fragment_order_gives_the_digits():
    """m16n8k32: A byte b of register 2 w + h (w: k half, h: row half) of lane
    (g, t) is row g + 8 h, k = 4 t + b + 16 w; B byte b of register w is
    column g, the same k.  Both sides place square _square(t, s, b, w) there,
    and a two-byte weight is low + 256 high."""
    rng = np.random.RandomState(1)
    assert sorted(_square(t, s, b, r) for t in range(4) for s in range(2) for b in range(4) for r in range(2)) == \
        list(range(64))
    cells = rng.randint(0, 3, (16, 64))
    lists = [rng.permutation(64)[:n] for n in (1, 5, 6, 7, 8, 9, 10, 11)]
    weight = np.zeros((64, 8), np.int64)
    for j, sq in enumerate(lists):
        weight[sq, j] = 3 ** np.arange(len(sq))
    # a position's words, shifted and masked, are the A registers
    p = [sum(int(c == 1) << i for i, c in enumerate(row)) for row in cells]
    o = [sum(int(c == 2) << i for i, c in enumerate(row)) for row in cells]
    d = np.zeros((2, 16, 8), np.int64)
    for s in range(2):
        a, b = np.zeros((16, 32), np.int64), np.zeros((2, 32, 8), np.int64)
        for t in range(4):
            for w in range(2):
                for row in range(16):
                    pw, ow = (p[row] >> (32 * w)) & 0xFFFFFFFF, (o[row] >> (32 * w)) & 0xFFFFFFFF
                    pw, ow = pw >> (2 * t), ((ow >> (2 * t)) << 1) & 0xFFFFFFFF
                    reg = ((pw >> s) & 0x01010101) | ((ow >> s) & 0x02020202)
                    for byte in range(4):
                        a[row, 16 * w + 4 * t + byte] = (reg >> (8 * byte)) & 255
                for byte in range(4):
                    wt = weight[_square(t, s, byte, w)]
                    b[0, 16 * w + 4 * t + byte], b[1, 16 * w + 4 * t + byte] = wt & 255, wt >> 8
        d += np.stack([a @ b[0], a @ b[1]])
    assert (weight >> 16 == 0).all()
    np.testing.assert_array_equal(d[0] + 256 * d[1], cells @ weight)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 8, 15, 32, 33, 255, 257, 8193])
@pytest.mark.parametrize("name", ["set5", "set8", "fixtures", "long", "many"])
def test_tile_indexer_at_its_edges(cuda, orc, n, name):
    masks = {"set5": SET5, "set8": SET8, "fixtures": list(FIXTURES.values()), "long": SET5 + LONG, "many": MANY}[name]
    pos = cb.generate_positions(7 + n, n, 0, 60)
    host = pos.cpu().numpy().view(np.uint64)
    for mode in ("reference", "expanded"):
        want = orc.group_index(masks, 0 if mode == "reference" else 1, host)
        g = cb.GroupIndexer(masks, mode)
        np.testing.assert_array_equal(g.indices(pos).cpu().numpy().view(np.uint32), want)
        # an output that no 8-byte store may be used on, and nothing past it
        k = g.nnz_per_row
        out = torch.full((n * k + 2,), -1, dtype=torch.int32, device="cuda")
        L.check(L.load().cas_index(g.handle, C.c_void_p(pos.data_ptr()), n, C.c_void_p(out[1:].data_ptr()),
                                   C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        got = out.cpu().numpy()
        np.testing.assert_array_equal(got[1:-1].view(np.uint32).reshape(n, k), want)
        assert got[0] == -1 and got[-1] == -1


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [[1, 5, 40, 31, 0, 7, 64], [16383, 2, 16385, 33]])
@pytest.mark.parametrize("mode", ["reference", "expanded"])
def test_blocked_indices_at_problem_bounds(cuda, orc, sizes, mode):
    """Rows of one warp step in several problems and blocks: the products read
    every index that was written."""
    n = sum(sizes)
    pos = cb.generate_positions(11, n, 0, 60)
    g = cb.GroupIndexer(SET8, mode)
    a = cb.MatrixCSR.from_positions_batched(g, pos, sizes)
    idx = orc.group_index(SET8, 0 if mode == "reference" else 1, pos.cpu().numpy().view(np.uint64)).astype(np.int64)
    cols = g.index_space_size
    idx += np.repeat(np.arange(len(sizes)), sizes)[:, None] * cols
    x = torch.randint(-8, 9, (cols * len(sizes),), device="cuda").double()  # integer sums: exact
    np.testing.assert_array_equal((a @ x).cpu().numpy(), x.cpu().numpy()[idx].sum(1))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 33, 255, 1025])
@pytest.mark.parametrize("name", ["set5", "one", "long"])
def test_tile_scores_at_their_edges(cuda, orc, n, name):
    """FP32 sums in slot order, one group of 16 slots and more, and variations
    too long for the tiles."""
    masks = {"set5": SET5, "one": SET5[:1], "long": SET5[3:] + [0x0F0F0F]}[name]
    g = cb.GroupIndexer(masks, "reference")
    w = np.random.RandomState(n).standard_normal((cb.estimator_stages(7), g.index_space_size)).astype(np.float32)
    pos = cb.generate_positions(5 + n, n, 0, 60)
    pos[0, 0] |= pos[0, 1] & -pos[0, 1]  # a square of both players (or a whole position, if it has none)
    host = pos.cpu().numpy().view(np.uint64)
    idx = orc.group_index(masks, 0, host)
    both = (host[:, 0] & host[:, 1]) != 0
    want = np.zeros(n, np.float32)
    empty = 64 - np.array([bin(int(p | o)).count("1") for p, o in host])
    for s in range(idx.shape[1]):
        ok = ~both
        want[ok] += w[empty[ok] // 7, idx[ok, s]]
    want[both] = np.nan
    got = cb.MultiStageScoreEstimator(masks, 7, w).eval(pos).cpu().numpy()
    np.testing.assert_array_equal(got, want)
