"""Batch scoring with as many pattern variations as an estimator takes
(cassandra_b200/csrc/estimator.cu): their tiles pass the shared memory that a
kernel has by default at 233 variations.  The FP32 sum in slot order, bitwise."""
import numpy as np
import pytest

import cassandra_b200 as cb

CORNERS = 0x8100000000000081  # one variation


def _masks(variations):
    """Short masks with this many variations in all: eight each, then one each."""
    eight = [m for m in range(1, 2048) if bin(m).count("1") in (2, 3, 4)
             and cb.GroupIndexer([m], "reference").nnz_per_row == 8][:variations // 8]
    masks = eight + [CORNERS] * (variations % 8)
    assert cb.GroupIndexer(masks, "reference").nnz_per_row == variations
    return masks


@pytest.mark.gpu
@pytest.mark.parametrize("variations", [231, 232, 233, 240, 241, 248, 255, 256])
@pytest.mark.parametrize("n", [1, 1000])
def test_scores_with_many_variations(cuda, orc, variations, n):
    masks = _masks(variations)
    cols = cb.GroupIndexer(masks, "reference").index_space_size
    w = np.random.RandomState(variations).standard_normal((cb.estimator_stages(10), cols)).astype(np.float32)
    pos = cb.generate_positions(variations + n, n, 0, 60)
    host = pos.cpu().numpy().view(np.uint64)
    idx = orc.group_index(masks, 0, host)
    stage = (64 - np.array([bin(int(p | o)).count("1") for p, o in host])) // 10
    want = np.zeros(n, np.float32)
    for s in range(idx.shape[1]):
        want += w[stage, idx[:, s]]
    got = cb.MultiStageScoreEstimator(masks, 10, w).eval(pos).cpu().numpy()
    np.testing.assert_array_equal(got, want)


@pytest.mark.gpu
def test_more_variations_are_refused(cuda):
    masks = _masks(256) + [CORNERS]
    cols = cb.GroupIndexer(masks, "reference").index_space_size
    with pytest.raises(cb.CasError):
        cb.MultiStageScoreEstimator(masks, 10, np.zeros((cb.estimator_stages(10), cols), np.float32))
