"""Folded packed networks (gates that hand on a row or a constant, and rows that nothing reads, taken out) against the oracle and
the layer-by-layer kernels: counts and rows."""
import numpy as np
import pytest
import torch

import difflogic_b200 as D
from difflogic_b200 import ops
from oracle import logic_oracle as O

pytestmark = pytest.mark.gpu

ALL = tuple(range(16))
# (rows of the input and of every layer, k, bytes of a row, word bits, gates): one gate kernel CTA and several, a remainder of the
# list's CTAs (256 neurons), layers of one row, classes of more neurons than a warp counts and classes of one, rows for each unit of the plain kernel (1, 2, 4, 8, 16 bytes), for the staged
# kernel (512 on) and a remainder of its column blocks (2048); classes counted with the last layer, in parts and apart; layers of
# which nothing is left, everything is, and of copies only (a value read many layers on)
CASES = [([5, 3, 4], 2, 16, 32, ALL), ([1, 1, 1, 1], 1, 3, 8, ALL), ([40, 257, 255, 256], 2, 6, 16, ALL), ([9, 70, 70], 7, 12, 32, ALL),
         ([300, 1001, 1001, 1001], 7, 24, 64, ALL), ([64, 3000, 500, 700], 1, 48, 64, ALL), ([64, 640, 640], 10, 512, 64, ALL),
         ([200, 4100, 4200], 2, 2064, 64, ALL), ([200] + 31 * [2050], 50, 528, 32, ALL), ([30, 400, 400, 400], 4, 1040, 64, (0, 15)),
         ([100, 40000, 40000], 1, 528, 64, ALL), ([64, 2500, 2600], 2, 4112, 64, ALL), ([20, 900, 900], 900, 1040, 64, ALL),
         ([64, 9000, 18002], 2, 4112, 64, ALL), ([30, 400, 400, 400], 4, 1040, 64, (3, 5, 10, 12)), ([100, 900, 900, 900], 9, 640, 64, (1, 2, 4, 6, 7, 8, 9, 11, 13, 14))]


@pytest.mark.parametrize("dims,k,row_bytes,bits,gates", CASES)
def test_counts_and_rows(dims, k, row_bytes, bits, gates):
    g = torch.Generator().manual_seed(row_bytes)
    layers = []
    for n_in, n_out in zip(dims[:-1], dims[1:]):
        a, b = torch.randint(0, n_in, (2, n_out), generator=g)
        b[:: 17] = a[:: 17]                                     # neurons that read one row twice
        layers.append((a, b, torch.tensor(gates, dtype=torch.uint8)[torch.randint(0, len(gates), (n_out,), generator=g)]))
    data = torch.randint(0, 256, (dims[0], row_bytes), generator=g, dtype=torch.uint8).numpy()
    x = torch.from_numpy(data.view("int%d" % bits))
    device_layers, xd = [tuple(t.cuda() for t in layer) for layer in layers], x.cuda()
    network = ops.FoldedLayers(dims[0], device_layers)
    left = network.program._dl_left
    assert len(left) == len(layers) and all(0 <= gates <= n for gates, n in zip(left[1:], dims[1:]))
    assert not network.rows if set(gates) <= {0, 3, 5, 10, 12, 15} else network.rows <= sum(dims[1:-1])
    rows = x.numpy()
    for a, b, gate in layers:
        rows = O.eval_packed(rows, a.numpy(), b.numpy(), gate.numpy())
    assert np.array_equal(ops.eval_folded(xd, network, row_bytes * 8).cpu().numpy(), rows)
    batch = row_bytes * 8 - 5
    one_by_one = xd
    for a, b, gate in device_layers:
        one_by_one = ops.eval_packed(one_by_one, a, b, gate)
    want = ops.groupbitsum(one_by_one, 5, k)
    packed = D.PackBitsTensor.from_packed(xd, 5)
    assert packed._folded_counts(network.sizes, network.rows, k) or row_bytes % 16 != 0
    if row_bytes % 16 == 0:
        assert torch.equal(ops.eval_folded(xd, network, batch, k), want)


# Rows longer than those that tail_counts_kernel takes: classes by the table of what is not constant, whole or in parts (more than 2040
# neurons), among them classes of constants only (some true, which are counted once) and of a few neurons.
@pytest.mark.parametrize("m", [700, 2040, 2100, 9001])
def test_classes_of_very_different_length(m):
    g, k, row_bytes = torch.Generator().manual_seed(m), 5, 4112
    dims = [64, 3000, k * m]
    layers = []
    for n_in, n_out in zip(dims[:-1], dims[1:]):
        a, b = torch.randint(0, n_in, (2, n_out), generator=g)
        layers.append([a, b, torch.randint(0, 16, (n_out,), generator=g).to(torch.uint8)])
    gate = layers[1][2].view(k, m)
    gate[1] = 15 * (gate[1] & 1)                            # constants only
    gate[2] = 0
    gate[3, 5:] = 15
    gate[4] = 6                                             # all needed
    layers[1][1] = (layers[1][0] + 1) % 3000
    x = torch.from_numpy(torch.randint(0, 256, (64, row_bytes), generator=g, dtype=torch.uint8).numpy().view("int64"))
    network, xd = ops.FoldedLayers(64, [tuple(t.cuda() for t in layer) for layer in layers]), x.cuda()
    rows = x.numpy()
    for a, b, gate in layers:
        rows = O.eval_packed(rows, a.numpy(), b.numpy(), gate.numpy())
    batch = row_bytes * 8 - 5
    want = np.concatenate([O.group_bit_sum(rows[c * m:(c + 1) * m], 5, 1) for c in range(k)], 1)
    for _ in range(2):
        assert np.array_equal(ops.eval_folded(xd, network, batch, k).cpu().numpy(), want)


def test_a_wide_network_is_folded(monkeypatch):
    """Through the modules: first pass, second pass, a pass with the output's rows, and one that finds no memory."""
    torch.manual_seed(6)
    model = torch.nn.Sequential(D.LogicLayer(70, 17000), D.LogicLayer(17000, 17000), D.LogicLayer(17000, 17000), D.GroupSum(10)).eval()
    layers = [m for m in model if isinstance(m, D.LogicLayer)]
    x = torch.rand(5001, 70, device="cuda") < 0.5
    want = O.packed_net_counts(x.cpu().numpy(), [l.indices[0].cpu() for l in layers], [l.indices[1].cpu() for l in layers],
                               [l.weights.detach().argmax(1).cpu().numpy().astype(np.uint8) for l in layers], 10, 32)
    folded = []
    run = ops.eval_folded
    monkeypatch.setattr(ops, "eval_folded", lambda *a: folded.append(a) or run(*a))

    def counts():
        with torch.no_grad():
            return model(D.PackBitsTensor(x)).cpu().numpy()
    assert np.array_equal(counts(), want) and not folded
    assert np.array_equal(counts(), want) and len(folded) == 1
    few = D.PackBitsTensor(x[:200])             # rows too short for the staged counting kernel
    assert np.array_equal(model[3](model[2](model[1](model[0](few)))).cpu().numpy(), want[:200]) and len(folded) == 2
    packed = D.PackBitsTensor(x)
    for layer in layers:
        packed = layer(packed)
    assert np.array_equal(ops.groupbitsum(packed.t, packed.pad_len, 10).cpu().numpy(), want) and len(folded) == 3

    def no_memory(*a):
        raise torch.cuda.OutOfMemoryError
    monkeypatch.setattr(ops, "eval_folded", no_memory)
    assert np.array_equal(counts(), want)
    with torch.no_grad():                       # nothing to fold: whole layers
        for layer in layers:
            layer.weights.zero_()
            layer.weights[:, 6] = 1.0
    monkeypatch.setattr(ops, "eval_folded", lambda *a: folded.append(a) or run(*a))
    first, again = counts(), counts()
    assert np.array_equal(first, again) and len(folded) == 3


@pytest.mark.parametrize("dims,k,both,route", [
    ([30, 600, 600, 16400], 10, False, ["folded"]),                          # the last layer does not fit the one kernel, gates fold
    ([30, 600, 600, 600, 16400], 10, True, ["one kernel", "with counts"]),   # they do not: the hidden layers go there
    ([30, 600, 600, 16400], 10, True, ["layer", "layer", "with counts"]),
    ([30, 17000, 17000, 17000], 10, True, ["layer", "layer", "with counts"]),    # nor do the hidden layers
    ([30, 2000, 2000, 2000], 2000, False, ["one kernel", "layer"]),          # the classes do not
    ([30, 2000, 2000, 2000], 2000, True, ["one kernel", "layer"])])
def test_where_networks_run_that_do_not_fit_the_one_kernel(monkeypatch, dims, k, both, route):
    """From the third pass on, and the counts of all passes."""
    torch.manual_seed(len(dims))
    model = torch.nn.Sequential(*[D.LogicLayer(*d) for d in zip(dims, dims[1:])], D.GroupSum(k)).eval()
    layers = list(model)[:-1]
    with torch.no_grad():
        if both:
            for layer in layers:
                kind = torch.tensor([1, 2, 4, 6, 7, 8, 9, 11, 13, 14], device="cuda")[torch.randint(0, 10, (layer.out_dim,), device="cuda")]
                layer.weights.zero_().scatter_(1, kind[:, None], 1.0)
                layer.set_connections(layer.indices[0], (layer.indices[0] + 1) % layer.in_dim)
        x = torch.rand(5001, dims[0], device="cuda") < 0.5
        want = O.packed_net_counts(x.cpu().numpy(), [l.indices[0].cpu() for l in layers], [l.indices[1].cpu() for l in layers],
                                   [l.weights.argmax(1).cpu().numpy().astype(np.uint8) for l in layers], k, 32)
        run = []
        for name, what in (("eval_folded", "folded"), ("eval_network", "one kernel"), ("eval_packed", "layer"), ("eval_groupbitsum", "with counts")):
            def spy(*a, kernel=getattr(ops, name), what=what, **kw):
                run.append(what)
                return kernel(*a, **kw)
            monkeypatch.setattr(ops, name, spy)
        for _ in range(4):
            del run[:]
            assert np.array_equal(model(D.PackBitsTensor(x)).cpu().numpy(), want)
    assert run == route
    if "folded" not in route and route[0] != "one kernel":      # built, found not to pay: nothing of it stays
        assert layers[-1]._folded_network.program == () and layers[-1]._folded_network.layer_by_layer == (max(dims[:-1]) > 16384)


def test_the_lists_are_all_that_stays():
    """17 bytes per neuron; what the sweeps need besides is given back."""
    layers = [tuple(t.cuda() for t in layer) for layer in _random_layers([100, 20000, 20000, 20000])]
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    network = ops.FoldedLayers(100, layers)
    assert network.program.numel() == 17 * 60000 and torch.cuda.memory_allocated() - before == -(-17 * 60000 // 512) * 512


def _random_layers(dims):
    g = torch.Generator().manual_seed(1)
    return [(*torch.randint(0, a, (2, b), generator=g), torch.randint(0, 16, (b,), generator=g).to(torch.uint8)) for a, b in zip(dims, dims[1:])]
