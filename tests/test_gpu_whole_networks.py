"""Networks that folding leaves as they are: every neuron evaluated, against the oracle and the folded evaluation."""
import numpy as np
import pytest
import torch

import difflogic_b200 as D
from difflogic_b200 import ops
from oracle import logic_oracle as O

pytestmark = pytest.mark.gpu

BOTH_INPUTS = [1, 2, 4, 6, 7, 8, 9, 11, 13, 14]     # gates that depend on both


def _layers(dims, gates, seed):
    g = torch.Generator().manual_seed(seed)
    layers = []
    for n_in, n_out in zip(dims[:-1], dims[1:]):
        a = torch.randint(0, n_in, (n_out,), generator=g)
        b = (a + 1 + torch.randint(0, n_in - 1, (n_out,), generator=g)) % n_in
        layers.append((a, b, gates(n_out, g).to(torch.uint8)))
    return layers


def _genuine(n, g):
    return torch.tensor(BOTH_INPUTS)[torch.randint(0, len(BOTH_INPUTS), (n,), generator=g)]


# every width of a row and number of threads: one CTA per SM and several, rows at the limit of a width, few and many classes
@pytest.mark.parametrize("dims,k,batch", [
    ([5, 3], 1, 1), ([40, 60, 60], 2, 100), ([784] + 4 * [8000], 10, 100), ([64, 16384, 16384], 2, 33), ([300, 1001, 1001], 7, 128),
    ([50, 640, 320, 640], 64, 7000), ([100, 10241, 10241], 11, 8 * 64 * 148), ([30, 10240, 10240], 10, 128 * 148 - 127),
    ([70] + 32 * [100], 100, 30001), ([117, 5000, 5120], 16, 50000), ([20, 12, 300], 300, 25000), ([33, 900, 990, 999], 999, 20),
    ([20, 4096, 4000], 10, 4 * 32 * 148), ([20, 8192, 8192], 1, 40000)])
def test_counts_and_rows(dims, k, batch):
    layers = _layers(dims, _genuine, batch)
    words = -(-batch // 128) * 2
    x = torch.randint(-2 ** 63, 2 ** 63 - 1, (dims[0], words), generator=torch.Generator().manual_seed(1))
    network = ops.NetworkProgram(dims[0], [tuple(t.cuda() for t in layer) for layer in layers])
    program, xd = network.program, x.cuda()
    assert program._dl_whole is not None
    rows, counts = ops.eval_network(xd, network, words * 64), ops.eval_network(xd, network, batch, k)
    hidden = x.numpy()
    for a, b, gate in layers:
        hidden = O.eval_packed(hidden, a.numpy(), b.numpy(), gate.numpy())
    assert np.array_equal(rows.cpu().numpy(), hidden)
    assert torch.equal(counts, ops.groupbitsum(rows, 0, k)[:batch])
    program._dl_whole = None
    assert torch.equal(ops.eval_network(xd, network, words * 64), rows) and torch.equal(ops.eval_network(xd, network, batch, k), counts)


@pytest.mark.parametrize("copies", [0, 99, 100, 101])
def test_line_between_the_two(copies):
    """At least three quarters of the neurons left as gates."""
    def gates(n, g):
        kinds = _genuine(n, g)
        kinds[:copies] = 3      # the first input
        return kinds
    program = ops.NetworkProgram(64, [tuple(t.cuda() for t in layer) for layer in _layers([64, 400], gates, copies)]).program
    assert int(program[3]) == 400 - copies and (program._dl_whole is not None) == (copies <= 100)


def test_through_the_layers(monkeypatch):
    """Counts for one number of classes and another, and rows, of a model whose passes are remembered: every pass runs the evaluation
    of all neurons."""
    torch.manual_seed(1)
    evaluate, programs = ops.eval_network, []
    monkeypatch.setattr(ops, "eval_network", lambda x, network, *a: programs.append(network.program) or evaluate(x, network, *a))
    model = [D.LogicLayer(30, 600), D.LogicLayer(600, 600)]
    with torch.no_grad():
        for layer in model:
            kind = torch.tensor(BOTH_INPUTS, device="cuda")[torch.randint(0, 10, (600,), device="cuda")]
            layer.weights.zero_().scatter_(1, kind[:, None], 1.0)
        x = torch.rand(1000, 30, device="cuda") < 0.5
        net = [layer.indices + (layer.weights.argmax(1).to(torch.uint8),) for layer in model]
        for k in (10, 10, 6, 10, 6):
            got = torch.nn.Sequential(*model, D.GroupSum(k)).eval()(D.PackBitsTensor(x))
            want = O.packed_net_counts(x.cpu().numpy(), *[[t[i].cpu() for t in net] for i in range(2)], [t[2].cpu().numpy() for t in net], k, 32)
            assert np.array_equal(got.cpu().numpy(), want)
        packed = model[1](model[0](D.PackBitsTensor(x)))
        assert np.array_equal(ops.groupbitsum(packed.t, packed.pad_len, 6).cpu().numpy(), want)
    # layers of 600 rows: built by the first pass; whoever changes k or reads rows finds the program there
    assert len(programs) == 6 and all(p is model[1]._network.program and p._dl_whole is not None for p in programs)


@pytest.mark.parametrize("fold", [True, False])
def test_small_passes_before_large_ones(monkeypatch, fold):
    """A small pass builds the program for all neurons, the first large one the folded network; the large form serves both then."""
    monkeypatch.setattr(ops, "FOLD_WORK", 2400 * 3000)
    torch.manual_seed(2)
    model = torch.nn.Sequential(D.LogicLayer(30, 2400), D.LogicLayer(2400, 2400), D.GroupSum(10)).eval()
    layers = list(model)[:-1]
    with torch.no_grad():
        if not fold:
            for layer in layers:
                layer.weights.zero_()
                layer.weights[:, 6] = 1.0
                layer.set_connections(layer.indices[0], (layer.indices[0] + 1) % layer.in_dim)
        x = torch.rand(5000, 30, device="cuda") < 0.5
        want = O.packed_net_counts(x.cpu().numpy(), [l.indices[0].cpu() for l in layers], [l.indices[1].cpu() for l in layers],
                                   [l.weights.argmax(1).cpu().numpy().astype(np.uint8) for l in layers], 10, 32)
        forms = []
        for n in (100, 100, 1400, 5000, 100, 5000):
            assert np.array_equal(model(D.PackBitsTensor(x[:n])).cpu().numpy(), want[:n])
            program = layers[1]._network.program
            forms.append("none" if program is None else "whole" if program._dl_whole is not None else "folded")
    assert forms == ["none"] + ["whole"] * 2 + ["folded" if fold else "whole"] * 3
