"""The generators wait for no stream but their own: targets are enqueued
(cassandra_b200/csrc/fit.cu), positions wait for the stream they run on.  A
bounded spin on another stream is still running when they return."""
import pytest
import torch

import cassandra_b200 as cb
from cassandra_b200 import _lib as L
from tests.golden.make_golden import SET5

pytestmark = pytest.mark.gpu

SPIN = 2_000_000_000  # cycles: about a second


def _matrix(rows):
    pos = cb.generate_positions(1, rows, 20, 40)
    return cb.MatrixCSR.from_positions(cb.GroupIndexer(SET5, "reference"), pos, "blocked")


def _while_spinning(call):
    """Whether the other stream's spin is still running after the calls."""
    call()  # every buffer is there
    torch.cuda.synchronize()
    other, done = torch.cuda.Stream(), torch.cuda.Event()
    with torch.cuda.stream(other):
        torch.cuda._sleep(SPIN)
        done.record()
    for _ in range(3):
        call()
    running = not done.query()
    torch.cuda.synchronize()
    return running


def test_targets_are_enqueued(cuda):
    a = _matrix(1000)
    want = cb.generate_targets(a, 3)
    assert _while_spinning(lambda: cb.generate_targets(a, 3))
    # and on the spinning stream itself: the call returns before its work is done
    side, done = torch.cuda.Stream(), torch.cuda.Event()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(SPIN)
        got = [cb.generate_targets(a, seed) for seed in (3, 4, 3)]
        done.record()
    assert not done.query()
    torch.cuda.synchronize()
    assert torch.equal(got[0], want) and torch.equal(got[2], want) and not torch.equal(got[1], want)


def test_positions_wait_for_their_own_stream_only(cuda):
    want = cb.generate_positions(5, 1000, 20, 40)
    assert _while_spinning(lambda: cb.generate_positions(5, 1000, 20, 40))
    assert torch.equal(cb.generate_positions(5, 1000, 20, 40), want)


def test_targets_under_capture(cuda):
    a = _matrix(1000)
    want = cb.generate_targets(a, 3)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = cb.generate_targets(a, 3)
    for _ in range(2):
        got.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)


def test_scratch_is_given_back(cuda):
    lib = L.load()
    a = _matrix(100)
    cb.generate_targets(a, 3)
    assert lib.cas_cached_memory() > 0
    lib.cas_release_cached_memory()
    assert lib.cas_cached_memory() == 0
    cb.generate_targets(a, 3)  # and works on
    torch.cuda.synchronize()
