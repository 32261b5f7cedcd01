"""The one-kernel evaluation of a packed network against the oracle and the layer-by-layer kernels: counts and rows."""
import copy
import ctypes

import numpy as np
import pytest
import torch

import difflogic_b200 as D
from difflogic_b200 import _native as N
from difflogic_b200 import ops
from oracle import logic_oracle as O

pytestmark = pytest.mark.gpu

# (rows of the input and of every layer, k, batch, bytes of a row per block): every block width, one and several CTAs per SM,
# one layer and the most there may be, layers of different widths, an odd number of rows, rows at the limit of a block width,
# classes shorter and longer than a warp's run of rows, the last block full, almost full and almost empty
CASES = [([5, 3], 1, 1, 4), ([40, 60, 60], 2, 100, 4), ([784] + 4 * [8000], 10, 100, 4), ([300, 1001, 1001], 7, 128, 4),
         ([64, 16384, 16384], 2, 33, 4), ([50, 640, 320, 640], 64, 7000, 8), ([100, 10241, 10241], 11, 8 * 64 * 148, 8),
         ([16384, 16384], 1, 40000, 8), ([30, 10240, 10240], 10, 128 * 148 - 127, 16), ([33, 2000, 2000, 999], 999, 20, 4),
         ([70] + 32 * [100], 100, 30001, 16), ([117, 5000, 5120], 16, 50000, 16), ([400, 2560, 2561], 13, 40001, 16),
         ([20, 12, 300], 300, 25000, 16)]


def _network(dims, seed):
    g = torch.Generator().manual_seed(seed)
    layers = []
    for n_in, n_out in zip(dims[:-1], dims[1:]):
        a, b = torch.randint(0, n_in, (2, n_out), generator=g)
        b[:: 17] = a[:: 17]                                     # neurons that read one row twice
        layers.append((a, b, (torch.arange(n_out) % 16)[torch.randperm(n_out, generator=g)].to(torch.uint8)))
    return layers


@pytest.mark.parametrize("dims,k,batch,width", CASES)
def test_counts_and_rows(dims, k, batch, width):
    layers = _network(dims, batch)
    words = -(-batch // 128) * 2
    g = torch.Generator().manual_seed(1)
    x = torch.randint(-2 ** 63, 2 ** 63 - 1, (dims[0], words), generator=g)
    device_layers = [tuple(t.cuda() for t in layer) for layer in layers]
    xd, sizes = x.cuda(), ops.network_sizes(dims[0], layers)
    assert N.lib().dl_eval_network_applicable(xd.data_ptr(), sizes, len(layers), words * 8, batch, k) == width
    network = ops.NetworkProgram(dims[0], device_layers)
    rows, hidden = xd, x.numpy()
    for (a, b, gate), (ha, hb, hg) in zip(device_layers, layers):
        rows = ops.eval_packed(rows, a, b, gate)
        hidden = O.eval_packed(hidden, ha.numpy(), hb.numpy(), hg.numpy())
    assert torch.equal(ops.eval_network(xd, network, words * 64), rows) and np.array_equal(rows.cpu().numpy(), hidden)
    counts = ops.eval_network(xd, network, batch, k)
    assert counts.shape == (batch, k) and counts.dtype == torch.int32
    want = ((hidden.view(np.uint64)[:, None, :] >> np.arange(64, dtype=np.uint64)[None, :, None]) & 1) if dims[-1] * words < 60000 else None
    if want is not None:
        want = want.transpose(0, 2, 1).reshape(k, dims[-1] // k, -1).sum(1).T[:batch]
        assert np.array_equal(counts.cpu().numpy(), want)
    assert torch.equal(counts, ops.groupbitsum(rows, words * 64 - batch, k) if words * 64 - batch < 64 else
                       ops.groupbitsum(rows, 0, k)[:batch])


def test_sizes_outside_the_range():
    x = torch.zeros(64, 4, dtype=torch.int64, device="cuda")

    def takes(dims, batch=256, k=1, x=x, row_bytes=32):
        return N.lib().dl_eval_network_applicable(x.data_ptr(), ops.network_sizes(dims[0], [(0, 0, torch.empty(n)) for n in dims[1:]]),
                                                  len(dims) - 1, row_bytes, batch, k)
    assert takes([64, 100])
    assert not takes([64, 16385]) and not takes([16385, 100]) and not takes([64] + 33 * [100]) and not takes([64])
    assert not takes([64, 100], k=3) and not takes([64, 100], k=0) and not takes([64, 100], batch=0) and not takes([64, 100], batch=257)
    assert not takes([64, 100], row_bytes=24) and not takes([64, 16384], k=16384)


def test_programs_follow_the_network():
    """A remembered program is not used for other gates, connections or layers, nor copied along with a layer."""
    torch.manual_seed(3)
    first, other, last = D.LogicLayer(50, 300), D.LogicLayer(50, 300), D.LogicLayer(300, 200)
    x = torch.rand(1000, 50, device="cuda") < 0.5

    def check(*layers):
        model = torch.nn.Sequential(*layers, D.GroupSum(10)).eval()
        h = x.cpu().numpy()
        with torch.no_grad():
            counts = model(D.PackBitsTensor(x))
            assert torch.equal(model(D.PackBitsTensor(x)), counts)
            packed = D.PackBitsTensor(x)
            for layer in layers:
                packed = layer(packed)
            assert torch.equal(ops.groupbitsum(packed.t, packed.pad_len, 10), counts)
        want = O.packed_net_counts(h, [l.indices[0].cpu() for l in layers], [l.indices[1].cpu() for l in layers],
                                   [l.weights.detach().argmax(1).cpu().numpy().astype(np.uint8) for l in layers], 10, 32)
        assert np.array_equal(counts.cpu().numpy(), want)

    check(first, last)
    check(other, last)
    check(first, last)
    with torch.no_grad():
        first.weights.copy_(first.weights[torch.randperm(300, device="cuda")])
    check(first, last)
    first.set_connections(*[i[torch.randperm(300, device="cuda")] for i in first.indices])
    check(first, last)
    last.indices[0].copy_(last.indices[0].flip(0))
    check(first, last)
    twin = copy.deepcopy(last)
    assert twin._network is None and last._network is not None
    check(first, twin)
    check(first)


def test_threads_with_networks_of_different_size():
    """Launches of one kernel with little and with much shared memory, from several threads at once: the limit that a launch sets is
    enough for the others'.  The entry point is called as directly as can be, so that calls of two threads overlap."""
    import threading
    failures = []
    start = threading.Barrier(4)

    def work(dims, k, batch):
        with torch.cuda.stream(torch.cuda.Stream()) as _:
            layers = [tuple(t.cuda() for t in layer) for layer in _network(dims, batch)]
            x = torch.randint(-2 ** 63, 2 ** 63 - 1, (dims[0], 2), generator=torch.Generator().manual_seed(1)).cuda()
            network = ops.NetworkProgram(dims[0], layers)
            want = ops.eval_network(x, network, batch, k)
            got = torch.empty_like(want)
            run = N.lib().dl_eval_network
            args = tuple(t(v) for t, v in zip(run.argtypes, (x.data_ptr(), network.program.data_ptr(), ctypes.addressof(network.sizes),
                                                             len(layers), got.data_ptr(), 0, 16, batch, k, N.stream_of(x))))
            start.wait()
            statuses = [run(*args) for _ in range(8000)]
            torch.cuda.current_stream().synchronize()
            if any(statuses) or not torch.equal(got, want):
                failures.append((dims, sum(map(bool, statuses))))
    threads = [threading.Thread(target=work, args=args) for args in 2 * [([64, 16384, 16384], 2, 33), ([40, 60, 60], 2, 100)]]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures


def test_threads_that_count_other_classes():
    """Two threads on streams of their own ask one network, whose program is there, for numbers of classes that it has not counted."""
    import threading
    dims, ks, batch = [100, 4800, 4800], (1, 2, 3, 4, 5, 6, 8, 10, 12, 15), 5000
    layers = _network(dims, batch)
    words = -(-batch // 128) * 2
    x = torch.randint(-2 ** 63, 2 ** 63 - 1, (dims[0], words), generator=torch.Generator().manual_seed(1))
    hidden = x.numpy()
    for a, b, gate in layers:
        hidden = O.eval_packed(hidden, a.numpy(), b.numpy(), gate.numpy())
    want = {k: O.group_bit_sum(hidden, 0, k)[:batch] for k in ks}
    xd, network = x.cuda(), ops.NetworkProgram(dims[0], [tuple(t.cuda() for t in layer) for layer in layers])
    torch.cuda.synchronize()
    start, got = threading.Barrier(2), [[], []]

    def work(mine, order):
        with torch.cuda.stream(torch.cuda.Stream()):
            for k in order:
                start.wait(60)
                got[mine].append((k, ops.eval_network(xd, network, batch, k)))
            torch.cuda.current_stream().synchronize()
    threads = [threading.Thread(target=work, args=args) for args in ((0, 3 * ks), (1, 3 * (ks[1:] + ks[:1])))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert [len(g) for g in got] == [30, 30]
    for k, counts in got[0] + got[1]:
        assert np.array_equal(counts.cpu().numpy(), want[k]), k


def test_a_graph_keeps_its_own_gates():
    torch.manual_seed(4)
    model = torch.nn.Sequential(D.LogicLayer(64, 320), D.LogicLayer(320, 320), D.GroupSum(10)).eval()
    x = torch.rand(640, 64, device="cuda") < 0.5
    with torch.no_grad():
        want = model(D.PackBitsTensor(x))
        graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=stream):
            counts = model(D.PackBitsTensor(x))
        graph.replay()
    assert torch.equal(counts, want)


def test_a_graph_outlives_the_gates_it_was_captured_with():
    """eval() again, other weights, an eager pass over them and allocations where freed gates would have been: the graph's counts
    stay those of the gates at its capture."""
    torch.manual_seed(5)
    model = torch.nn.Sequential(D.LogicLayer(64, 320), D.LogicLayer(320, 320), D.GroupSum(10)).eval()
    x = torch.rand(640, 64, device="cuda") < 0.5
    with torch.no_grad():
        want = model(D.PackBitsTensor(x)).clone()
        graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=stream):
            counts = model(D.PackBitsTensor(x))
        for change in range(3):
            if change == 1:
                model.train()
            model.eval()
            if change == 2:
                for layer in model[:2]:
                    layer.weights.copy_(layer.weights.flip(1))
            for _ in range(3):
                now = model(D.PackBitsTensor(x))
            over = [torch.full((320,), 7, dtype=torch.uint8, device="cuda") for _ in range(64)]
            counts.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(counts, want) and torch.equal(now, want) == (change < 2) and len(over) == 64
