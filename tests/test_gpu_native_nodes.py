"""The native autograd nodes against the Python functions that take what they leave: same bits, same refusals."""
import types

import pytest
import torch

import difflogic_b200 as D
from difflogic_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.fixture
def python_nodes(monkeypatch):
    """Switches the native nodes off for the rest of the test when called."""
    return lambda: monkeypatch.setattr(N, "nodes", lambda: types.SimpleNamespace(layer=lambda *a: None, group_sum=lambda *a: None))


def _net(n_in, width, k):
    torch.manual_seed(n_in)
    return torch.nn.Sequential(D.LogicLayer(n_in, width, grad_factor=2.0), D.LogicLayer(width, width), D.GroupSum(k, tau=3.0))


# one sample, an odd batch, whole 16-byte rows; 12000 neurons and 2e6 outputs: the walk kernels, complete and not, whole units and not
SIZES = [(5, 3, 1, 1), (64, 320, 10, 61), (117, 640, 10, 100), (12000, 12000, 4, 168), (12000, 12000, 2, 169), (100, 12000, 3, 172)]
INPUTS = {"batch major": lambda x: x, "feature major": lambda x: x.t().contiguous().t(), "strided": lambda x: torch.stack([x, x], 2)[:, :, 0]}


@pytest.mark.parametrize("layout", list(INPUTS))
@pytest.mark.parametrize("grad_x", [False, True])
@pytest.mark.parametrize("n_in,width,k,batch", SIZES)
def test_same_bits(python_nodes, n_in, width, k, batch, grad_x, layout):
    model = _net(n_in, width, k)
    x = INPUTS[layout](torch.rand(batch, n_in, device="cuda")).requires_grad_(grad_x)
    y = torch.randint(0, k, (batch,), device="cuda")

    def run():
        x.grad = None
        model.zero_grad()
        h = model[0](x)
        scores = model[2](model[1](h))
        torch.nn.functional.cross_entropy(scores, y).backward()
        return [h.detach(), scores.detach(), x.grad] + [p.grad for p in model.parameters()]
    before = N.nodes().launches()
    native = run()
    # per layer forward, weight gradient and, unless both come from one kernel, input gradient; both ways of GroupSum
    assert N.nodes().launches() - before >= 6
    python_nodes()
    for a, b in zip(native, run()):
        assert (a is None and b is None) or (torch.equal(a, b) and (batch == 1 or a.stride() == b.stride()))


def test_hooks_for_saved_tensors_and_changed_weights():
    model, x = _net(64, 320, 10), torch.rand(33, 64, device="cuda")
    model(x).sum().backward()
    want = [p.grad.clone() for p in model.parameters()]
    model.zero_grad()
    with torch.autograd.graph.save_on_cpu():
        out = model(x)
    out.sum().backward()
    assert all(torch.equal(p.grad, w) for p, w in zip(model.parameters(), want))
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.double() if t.is_floating_point() else t, lambda t: t):
        out = model(x)
    with pytest.raises(RuntimeError):
        out.sum().backward()
    out = model(x)
    with torch.no_grad():
        model[0].weights.add_(1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.sum().backward()


@pytest.mark.parametrize("native", [True, False])
def test_what_is_refused(python_nodes, native):
    if not native:
        python_nodes()
    layer, x = D.LogicLayer(64, 320), torch.rand(33, 64, device="cuda")
    for wrong, error in ((x.double(), RuntimeError), (x[:, :63], AssertionError), (x[0], AssertionError), (x.cpu(), AssertionError)):
        with pytest.raises(error):
            layer(wrong)
    with pytest.raises(RuntimeError):
        torch.func.vmap(layer)(x[None])
    with pytest.raises(RuntimeError):
        torch.func.jvp(layer, (x,), (x,))
    with torch.autograd.forward_ad.dual_level(), pytest.raises(RuntimeError):
        x = x.t().contiguous().t()
        layer(torch.autograd.forward_ad.make_dual(x, x))
    h = layer(x)
    h.mul_(2.0)                       # an output may be written to
    h.sum().backward()
    with torch.no_grad():
        assert not layer(x).requires_grad


def test_an_optimizer_switched_on_between_the_passes():
    """FlatAdam stepping inside backward is asked for when the backward pass runs."""
    from difflogic_b200.optim import FlatAdam
    model, x = _net(64, 320, 10), torch.rand(33, 64, device="cuda")
    opt = FlatAdam(model.parameters(), lr=0.01)
    start = opt.flat_param.clone()
    out = model(x)
    opt.enable_step_in_backward(True)
    out.square().sum().backward()
    opt.enable_step_in_backward(False)
    assert all(p.grad is None for p in model.parameters()) and not torch.equal(opt.flat_param, start)
