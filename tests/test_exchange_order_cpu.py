"""Which events the launch of a bucket's exchange waits for (FlatAdam), with streams, events and kernels replaced by stand-ins: a
bucket's gradients may be written on several streams."""
import types

import pytest
import torch

from difflogic_b200 import _native as N
from difflogic_b200.optim import FlatAdam


class _Stream:
    def __init__(self, handle):
        self.cuda_stream, self.queue = handle, []

    def wait_event(self, event):
        self.queue.append(("wait", event.of))


class _Event:
    def record(self, stream):
        self.of = tuple(stream.queue)          # what is complete once the event is


class _Device:
    def __init__(self, *a):
        pass

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        return False


@pytest.fixture
def world(monkeypatch):
    w = types.SimpleNamespace(main=_Stream(1), side=_Stream(2), comm=_Stream(3), launches=[])
    w.current = w.main
    by_handle = {s.cuda_stream: s for s in (w.main, w.side, w.comm)}

    def launch(*args):
        *_, how, handle = args
        stream = by_handle[handle]
        known = set()

        def reach(queue):
            for kind, what in queue:
                known.add(what) if kind == "kernel" else reach(what)
        reach(stream.queue)
        w.launches.append((known, how, stream))
        stream.queue.append(("kernel", "exchange"))
        return 0
    monkeypatch.setattr(N, "lib", lambda: types.SimpleNamespace(dl_exchange_packets_f32=launch, dl_exchange_bucket_f32=launch))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: w.current)
    monkeypatch.setattr(torch.cuda, "Event", _Event)
    monkeypatch.setattr(torch.cuda, "device", _Device)
    return w


def _optimizer(world, count, buckets, packets):
    opt = object.__new__(FlatAdam)
    params = [torch.zeros(16) for _ in range(count)]
    opt._params = params
    opt._slices = {p: (16 * i, 16) for i, p in enumerate(params)}
    opt._plan_exchange_buckets(buckets)
    opt.flat_param = opt.flat_grad = opt.exp_avg = opt.exp_avg_sq = torch.zeros(16 * count)
    opt.state_t = torch.zeros(len(opt._buckets), 16, dtype=torch.int32)
    opt.param_groups = [dict(lr=0.1, betas=(0.9, 0.999), eps=1e-8)]
    opt._exchange, opt._packet_form, opt._one_pass, opt._forms_fixed = (0, 2), set(range(len(opt._buckets))) if packets else set(), set(), False
    opt._one_pass_bytes, opt._wait_limit_us, opt._announce_in_backward, opt._push_in_backward = 0, 0, False, False
    opt._peer_ptrs = dict(grad_inbox=None, param_inbox=None, param=None, grad=None, flags=None)
    opt._inbox_off, opt._inbox_stride, opt._comm_streams, opt.exchange_enabled = [0] * len(opt._buckets), 1, [world.comm], True
    opt._begin_exchange_step()
    return opt


def _gradients(world, opt, streams):
    """Queues the gradient kernel of every parameter, the last layer's first, each on the stream named for it."""
    for i in reversed(range(len(streams))):
        world.current = stream = getattr(world, streams[i])
        stream.queue.append(("kernel", "gradient %d" % i))
        opt.gradient_queued(opt._params[i])
    world.current = world.main


@pytest.mark.parametrize("packets", [False, True])
@pytest.mark.parametrize("buckets", [1, 2, 4])
@pytest.mark.parametrize("streams", [("main",) * 4, ("main", "side", "side", "side"), ("main", "side", "main", "side"),
                                     ("side", "main", "side", "main"), ("side", "side", "main", "main")])
def test_an_exchange_starts_after_all_gradients_of_its_bucket(world, streams, buckets, packets):
    opt = _optimizer(world, 4, buckets, packets)
    for step in range(2):
        world.launches.clear()
        for s in (world.main, world.side, world.comm):
            s.queue.clear()
        _gradients(world, opt, streams)
        assert len(world.launches) == len(opt._buckets)
        for (known, how, stream), (_, _, group) in zip(world.launches, reversed(opt._buckets)):
            mine = [i for i, p in enumerate(opt._params) if any(p is q for q in group)]
            assert {"gradient %d" % i for i in mine} <= known
            # the set-up may overlap the kernel in front only where that is the last thing waited for
            alone = len({streams[i] for i in mine}) == 1
            assert how == (N.LAUNCH_OVERLAP_SETUP if stream is not world.comm and alone else N.LAUNCH_PLAIN)
        opt._begin_exchange_step()
