"""Evaluator ranges on both sides of the rows that are resident at once
(cassandra_b200/csrc/fast.cu: how far ahead a row's index words are loaded):
scores exact on integer-valued weights, the loss of a training step and the
gradient behind its first moment against 64 bits."""
import pytest
import torch

import cassandra_b200 as cb
from cassandra_b200.evaluator import EvaluatorFunction, PatternEvaluator, Trainer
from tests.golden.make_golden import SET5, SET8

pytestmark = pytest.mark.gpu

RESIDENT = 7 * 128  # rows per SM
TWELVE = SET8 + [0xC3, 0x0303, 0x81, 0x1818]  # more patterns than words are held of; slots 8, 4, 2 and 1


def _sizes():
    bound = RESIDENT * torch.cuda.get_device_properties(0).multi_processor_count
    return [1, 127, 129, bound - 1, bound, bound + 1, 600_001]


@pytest.mark.parametrize("name,mode", [("set8", "expanded"), ("set5", "reference"), ("twelve", "reference"),
                                       ("twelve", "expanded")])
def test_scores(cuda, name, mode):
    masks = {"set8": SET8, "set5": SET5, "twelve": TWELVE}[name]
    sizes = _sizes()
    pos = cb.generate_positions(1, max(sizes) + 3, 10, 50)
    model = PatternEvaluator(masks, pos, mode)
    w = torch.randint(-8, 9, (model.indexer.index_space_size,), device="cuda").float()
    want = w[model.indexer.indices(pos).long()].sum(1)
    for n in sizes:
        for row0 in (0, 3):
            assert torch.equal(EvaluatorFunction.apply(w, model.csr, row0, row0 + n), want[row0:row0 + n])


@pytest.mark.parametrize("name,mode", [("set8", "expanded"), ("set5", "reference")])
@pytest.mark.parametrize("which", range(7))
def test_loss_and_gradient(cuda, name, mode, which):
    n = _sizes()[which]
    pos = cb.generate_positions(2, n, 10, 50)
    model = PatternEvaluator(SET8 if name == "set8" else SET5, pos, mode)
    target = torch.randint(-20, 21, (n,), device="cuda").float()
    t = Trainer(model, target, batch=2 * n + 32768, l2=0.0, delta=4.0)
    w = torch.randint(-2, 3, (model.indexer.index_space_size,), device="cuda").float()
    with torch.no_grad():
        model.weight.copy_(w)
    loss = t.epoch()
    idx = model.indexer.indices(pos).long()
    d = (w.double()[idx].sum(1) - target.double())
    # every row's loss is exact in FP32, their sum is FP64
    want = torch.nn.functional.huber_loss(d, torch.zeros_like(d), delta=4.0)
    assert abs(loss - float(want)) <= 1e-12 * (1 + float(want))
    ds = d.clamp(-4, 4) / n
    grad = torch.zeros(w.numel(), dtype=torch.float64, device="cuda")
    size = torch.zeros_like(grad)
    for to, v in ((grad, ds), (size, ds.abs())):
        to.index_add_(0, idx.flatten(), v.repeat_interleave(idx.shape[1]))
    # m = 0.1 g; an FP32 sum of at most 32 entries a lane, its scan, and a
    # partial per round of 1,024 and per block: (n / 32 + 64) roundings at most
    err = (t._m.double() / float(torch.tensor(1.0) - torch.tensor(0.9)) - grad).abs()
    assert bool((err <= (n / 32 + 64) * 2.0**-24 * size).all())
