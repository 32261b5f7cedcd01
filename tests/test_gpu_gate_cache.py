"""The arg-max gates that packed inference works from follow the weights through every way the package has of updating them."""
import pytest
import torch

import difflogic_b200 as D
from difflogic_b200.optim import FlatAdam
from difflogic_b200.training import TrainStep

pytestmark = pytest.mark.gpu


def _counts(model, xb):
    model.eval()
    with torch.no_grad():
        counts = model(D.PackBitsTensor(xb, bit_count=32))
        assert torch.equal(model(D.PackBitsTensor(xb, bit_count=32)), counts)         # the second pass, by whichever kernels
    # the same network from scratch: nothing remembered
    fresh = [(l.weights.detach().argmax(1), l.indices) for l in model if isinstance(l, D.LogicLayer)]
    h = xb
    for gate, (a, b) in fresh:
        A, B = h[:, a], h[:, b]
        bits = [(gate >> s) & 1 for s in (3, 2, 1, 0)]
        h = torch.where(A, torch.where(B, bits[3].bool(), bits[2].bool()), torch.where(B, bits[1].bool(), bits[0].bool()))
    want = h.reshape(h.shape[0], model[-1].k, -1).sum(-1).int()
    assert torch.equal(counts, want)
    return counts


@pytest.mark.parametrize("way", ["loop", "step", "captured", "replay without train()"])
def test_gates_follow_the_optimizer(way):
    torch.manual_seed(0)
    model = torch.nn.Sequential(D.LogicLayer(64, 200), D.LogicLayer(200, 200), D.GroupSum(10, 3.0))
    opt = FlatAdam(model.parameters(), lr=1.0)     # large steps: the arg-max of most neurons moves
    x = (torch.rand(40, 64, device="cuda") < 0.4).float()
    y = torch.randint(0, 10, (40,), device="cuda")
    xb = x.bool()
    step = None
    if way != "loop":
        step = TrainStep(model, opt)
        if way != "step":
            step.capture(x, y)
    before = _counts(model, xb)
    if way != "replay without train()":
        model.train()
    for _ in range(3):
        if way == "loop":
            torch.nn.functional.cross_entropy(model(x), y).backward()
            opt.step()
            opt.zero_grad()
        elif way == "replay without train()":
            step.replay()
        else:
            step(x, y)
    after = _counts(model, xb)
    assert not torch.equal(before, after)


@pytest.mark.parametrize("way", ["loop", "captured"])
def test_an_update_leaves_earlier_graphs_usable(way):
    """The optimizer's kernels change the weights in place without autograd's version counters: a loss computed before a step can
    be differentiated after it."""
    torch.manual_seed(1)
    model = torch.nn.Sequential(D.LogicLayer(64, 200), D.LogicLayer(200, 200), D.GroupSum(10, 3.0))
    opt = FlatAdam(model.parameters(), lr=0.01)
    x, y = (torch.rand(40, 64, device="cuda") < 0.4).float(), torch.randint(0, 10, (40,), device="cuda")
    step = TrainStep(model, opt).capture(x, y) if way == "captured" else None
    versions = [p._version for p in model.parameters()]
    loss = torch.nn.functional.cross_entropy(model(x), y)
    if way == "loop":
        loss.backward(retain_graph=True)
        opt.step()
    else:
        step.replay()
    opt.zero_grad()
    loss.backward()
    assert all(p.grad is not None and bool(torch.isfinite(p.grad).all()) for p in model.parameters())
    assert versions == [p._version for p in model.parameters()]
