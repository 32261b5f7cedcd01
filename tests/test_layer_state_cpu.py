"""What a LogicLayer derives from its weights and connections and keeps (arg-max gates, the walk, the packed network's program),
with the kernels replaced by stand-ins: when it is made anew, how long it lives, what a captured graph may rely on."""
import weakref

import pytest
import torch

import difflogic_b200 as D
from difflogic_b200 import ops


class _Cuda:
    """Stand-in for the state of torch.cuda that the code under test asks for."""
    def __init__(self, monkeypatch):
        self.capturing = False
        monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: self.capturing)
        stream = type("Stream", (), {"synchronize": lambda s: None, "record_event": lambda s: "event"})()
        monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: stream)
        monkeypatch.setattr(torch.cuda, "synchronize", lambda device=None: None)


@pytest.fixture
def cuda(monkeypatch):
    return _Cuda(monkeypatch)


def _layer(n_in=8, n_out=8):
    return D.LogicLayer(n_in, n_out, device="cpu", implementation="cuda").eval()


@pytest.fixture
def argmax(monkeypatch):
    made = []

    def gates(w):
        made.append(w.argmax(-1).to(torch.uint8))
        return made[-1]
    monkeypatch.setattr(ops, "argmax_gates", gates)
    return made


def test_gates_stay_while_the_mode_stays(cuda, argmax):
    layer = _layer()
    kept = weakref.ref(layer._gate_ids())
    argmax.clear()
    layer.eval()
    assert kept() is not None and layer._gate_ids() is kept() and not argmax
    layer.train()
    layer.eval()
    layer._gate_ids()
    assert len(argmax) == 1


def test_gates_that_a_graph_reads_live_as_long_as_the_layer(cuda, argmax):
    layer = _layer()
    layer._gate_ids()
    cuda.capturing = True
    read = weakref.ref(layer._gate_ids())
    cuda.capturing = False
    argmax.clear()
    layer.train()
    layer.eval()
    with torch.no_grad():
        layer.weights.add_(1.0)
    assert layer._gate_ids() is not read() and read() is not None
    del layer
    argmax.clear()
    assert read() is None


@pytest.mark.parametrize("rows", [False, True])
def test_layers_applied_before_a_capture_that_runs_them(cuda, argmax, monkeypatch, rows):
    """A packed layer runs when its output is wanted: a capture may begin in between, and its graph reads the gates."""
    monkeypatch.setattr(ops, "eval_network_applicable", lambda x, sizes, batch, k: True)
    monkeypatch.setattr(ops, "eval_packed", lambda x, a, b, gate: x)
    monkeypatch.setattr(ops, "eval_groupbitsum_parts_applicable", lambda x, n_out, k: False)
    monkeypatch.setattr(ops, "eval_groupbitsum_applicable", lambda x, n_out, k: False)
    monkeypatch.setattr(ops, "groupbitsum", lambda x, pad_len, k, padded: "counts")
    layers = [_layer(), _layer()]
    packed = D.PackBitsTensor.from_packed(torch.ones(8, 2, dtype=torch.int32), 0)
    for layer in layers:
        packed._push_layer(layer)
    read = [weakref.ref(gate) for _, gate in packed._pending]
    cuda.capturing = True
    assert packed.t is not None if rows else packed.group_sum(2) == "counts"
    cuda.capturing = False
    del packed
    argmax.clear()
    for layer in layers:
        layer.train()
    assert all(gate() is not None for gate in read) and all(layer._network is None for layer in layers)


def test_gates_that_only_a_graph_computes_are_not_used_outside_it(cuda, argmax):
    layer = _layer()
    cuda.capturing = True
    inside = layer._gate_ids()
    cuda.capturing = False
    assert layer._gate_ids() is not inside


def test_gates_follow_updates_that_autograd_does_not_see(cuda, argmax):
    from difflogic_b200.optim import count_update
    layer = _layer()
    layer._gate_ids()
    version = layer.weights._version
    layer.weights.data.copy_(layer.weights.data.flip(1))     # as a kernel does: past the version counter
    count_update([layer.weights])
    assert torch.equal(layer._gate_ids(), layer.weights.argmax(-1).to(torch.uint8)) and layer.weights._version == version


@pytest.fixture
def walks(monkeypatch):
    """build_walk keeps what it was built from in place of the entries."""
    made = []

    def build(a, b, n_in):
        made.append((torch.stack([a, b]), True))
        return made[-1]
    monkeypatch.setattr(ops, "build_walk", build)
    return made


def test_a_walk_is_that_of_the_connections(cuda, walks):
    layer = _layer(12000, 12000).train()

    def check():
        assert torch.equal(layer._walk_for(1000)[0], torch.stack(layer.indices))
    check()
    check()
    assert len(walks) == 1
    layer.indices[0].copy_(layer.indices[0].flip(0))
    check()
    layer.indices = (layer.indices[0], layer.indices[1].flip(0))
    check()
    layer.indices = tuple(i.clone() for i in layer.indices)
    check()
    assert len(walks) == 4
    layer.set_connections(layer.indices[1], layer.indices[0])
    check()


def test_a_capture_takes_no_walk_of_other_connections(cuda, walks):
    layer = _layer(12000, 12000).train()
    cuda.capturing = True
    assert layer._walk_for(1000) is None          # none yet, and none is built
    cuda.capturing = False
    layer._walk_for(1000)
    cuda.capturing = True
    walks.clear()
    entries = weakref.ref(layer._walk_for(1000)[0])
    layer.indices[0].copy_(layer.indices[0].flip(0))
    assert layer._walk_for(1000) is None
    cuda.capturing = False
    layer._walk_for(1000)
    assert entries() is not None                  # the graph reads it


class _OnCuda:
    """What the checks of ops ask of a CUDA tensor, and nothing that could be launched."""
    is_cuda = True

    def __init__(self, rows, columns, dtype=torch.float32):
        self.shape, self.dtype = (rows, columns), dtype

    def dim(self):
        return 2

    def is_contiguous(self):
        return True


def test_walks_are_refused_for_other_rows(monkeypatch):
    """A walk's entries are row numbers; the gather kernels' index vectors are refused when they do not fit the weights."""
    from difflogic_b200 import _native

    def launched(*a):
        raise AssertionError("went on to launch")
    monkeypatch.setattr(_native, "on_device", launched)
    monkeypatch.setattr(_OnCuda, "new_empty", lambda self, shape: launched(), raising=False)
    walk = ops.Walk(None, True, 20, 30)
    for n_in, n_out in ((20, 29), (20, 31), (19, 30)):
        x, w, gy, coef = _OnCuda(n_in, 8), _OnCuda(n_out, 16), _OnCuda(n_out, 8), _OnCuda(n_out, 4)
        with pytest.raises(RuntimeError, match="rows"):
            ops.logic_forward_walk(x, w, walk)
        with pytest.raises(RuntimeError, match="rows"):
            ops.logic_backward_walk(x, gy, coef, w, walk, want_grad_x=False)


def test_a_walk_is_built_of_int64_vectors_only():
    """dl_build_walk reads host copies of them as int64."""
    class Index(_OnCuda):
        def dim(self):
            return 1

        def numel(self):
            return 4

        def cpu(self):
            raise AssertionError("went on to build")
    with pytest.raises(RuntimeError, match="int64"):
        ops.build_walk(Index(4, 1, torch.int32), Index(4, 1, torch.int32), 4)


def test_one_pass_in_eval_mode_builds_no_walk(cuda, walks):
    layer = _layer(12000, 12000)
    assert layer._walk_for(1000) is None and not walks
    assert layer._walk_for(1000) is not None and len(walks) == 1
    layer.indices[0].copy_(layer.indices[0].flip(0))         # other connections: from the start again
    assert layer._walk_for(1000) is None and len(walks) == 1
    assert layer.train()._walk_for(1000) is not None and len(walks) == 2
    assert layer.eval()._walk_for(1000) is not None and len(walks) == 2
    assert layer._walk_for(10) is None


def test_connections_made_in_inference_mode(cuda, walks, argmax, monkeypatch):
    """They have no version counter, so that nothing is kept for them: a layer of such connections (a model moved to the GPU in
    inference mode) runs the kernels that read them on every call."""
    with torch.inference_mode():
        layer = _layer(12000, 12000)
        layer.indices = tuple(i.clone() for i in layer.indices)
    for mode in (layer.eval, layer.train, layer.eval):
        mode()
        for _ in range(3):
            assert layer._walk_for(1000) is None and not walks
    monkeypatch.setattr(ops, "eval_network_applicable", lambda x, sizes, batch, k: True)
    monkeypatch.setattr(ops, "eval_packed", lambda x, a, b, gate: x[a] & x[b])
    for _ in range(3):
        packed = D.PackBitsTensor.from_packed(torch.ones(12000, 2, dtype=torch.int32), 0)
        packed._pending = [(layer, torch.zeros(12000, dtype=torch.uint8))] * 2
        assert packed.t.shape == (12000, 2)


def test_a_program_is_built_for_the_second_pass(cuda, argmax, monkeypatch):
    """A batch by single layers takes less time than building the program: one pass over a set of weights builds none."""
    built, single = [], []

    def build(network):
        built.append(network)
        assert network.gates_ready == "event"
        network.program = torch.zeros(1)
    monkeypatch.setattr(ops, "_index", lambda t, name, n=None: None)
    monkeypatch.setattr(ops.N, "on_device", lambda t: ops.N._ALREADY_THERE)
    monkeypatch.setattr(ops.NetworkProgram, "build", build)
    monkeypatch.setattr(ops, "eval_network_applicable", lambda x, sizes, batch, k: True)
    monkeypatch.setattr(ops, "eval_network", lambda x, network, batch, k=None: x if k is None else "counts")
    monkeypatch.setattr(ops, "eval_groupbitsum_parts_applicable", lambda x, n_out, k: False)
    monkeypatch.setattr(ops, "eval_groupbitsum_applicable", lambda x, n_out, k: False)
    monkeypatch.setattr(ops, "groupbitsum", lambda x, pad_len, k, padded: "counts")

    def eval_packed(x, a, b, gate):
        single.append(gate)
        return x
    monkeypatch.setattr(ops, "eval_packed", eval_packed)
    monkeypatch.setattr(D.packbitstensor, "PROGRAM_AT_ONCE_ROWS", 7)
    layers = [_layer() for _ in range(4)]

    def passes(model, *, rows=False):
        """(layers run one by one, programs built) in one pass."""
        del built[:], single[:]
        packed = D.PackBitsTensor.from_packed(torch.ones(8, 2, dtype=torch.int32), 0)
        for layer in model:
            packed._push_layer(layer)
        assert packed.t is not None if rows else packed.group_sum(2) == "counts"
        return len(single), len(built)

    for rows in (False, True):
        for layer in layers:
            layer.train()
            layer.eval()
        assert [passes(layers, rows=rows) for _ in range(3)] == [(4, 0), (0, 1), (0, 0)]
        with torch.no_grad():
            layers[1].weights.add_(1.0)
        assert [passes(layers, rows=rows) for _ in range(3)] == [(4, 0), (0, 1), (0, 0)]
        layers[2].indices[0].copy_(layers[2].indices[0].flip(0))
        assert [passes(layers, rows=rows) for _ in range(3)] == [(4, 0), (0, 1), (0, 0)]
        cuda.capturing = True
        assert passes(layers, rows=rows) == (4, 0)
        cuda.capturing = False
        assert passes(layers, rows=rows) == (0, 0)
    assert layers[2]._network is None                     # nothing is noted for a part of the network
    for limit, value in (("ROWS", 8), ("SAMPLES", 64)):   # a narrow network, a large batch: the first pass builds it
        monkeypatch.setattr(D.packbitstensor, "PROGRAM_AT_ONCE_ROWS", 7)
        monkeypatch.setattr(D.packbitstensor, "PROGRAM_AT_ONCE_" + limit, value)
        for layer in layers:
            layer.train()
            layer.eval()
        assert [passes(layers) for _ in range(2)] == [(0, 1), (0, 0)]


@pytest.mark.parametrize("kind", [ops.NetworkProgram, ops.FoldedLayers])
def test_tables_are_seen_when_they_are_finished(cuda, monkeypatch, kind):
    """Threads share a program's class tables, and a thread that finds one launches on a stream that waits for nothing."""
    monkeypatch.setattr(ops.N, "on_device", lambda t: ops.N._ALREADY_THERE)
    monkeypatch.setattr(ops.N, "stream_of", lambda t: 7)
    network, program = kind.__new__(kind), torch.zeros(4, dtype=torch.int32)
    network.sizes, network.layers, network.counted = (8, 8, 8), [()] * 2, 2
    program._dl_tables, seen = {}, []
    monkeypatch.setattr(kind, "_table_of", lambda network, program, k, stream: torch.zeros(1))
    stream = torch.cuda.current_stream()
    monkeypatch.setattr(type(stream), "synchronize", lambda stream: seen.append(set(program._dl_tables)))
    for k in (1, 2, 4, 8, 1):                             # by reading rows first, then counting; by counting with other classes
        table = network.table(program, k)
        assert program._dl_tables[k] is table and table._dl_stream == 7
    assert seen == [set(), {1}, {1, 2}, {1, 2, 4}]
    network.table(program, 16)                            # a fifth: from the start again
    assert seen[4:] == [{1, 2, 4, 8}] and set(program._dl_tables) == {16}


def test_a_table_is_that_of_the_classes_it_is_kept_under(cuda, monkeypatch):
    """`counted` is what the latest pass asks for; another thread may change it while one builds."""
    network = ops.NetworkProgram.__new__(ops.NetworkProgram)
    network.sizes, network.layers, network.counted, made = (8, 8, 8), [(None, None, torch.zeros(8))] * 2, 2, []
    words = type("Library", (), {"dl_network_program_words": lambda s, sizes, n: 8, "dl_network_fold": None, "dl_network_order": lambda *a: 0})()
    monkeypatch.setattr(ops.N, "lib", lambda: words)
    monkeypatch.setattr(ops.N, "on_device", lambda t: ops.N._ALREADY_THERE)
    monkeypatch.setattr(ops.N, "stream_of", lambda t: 7)
    monkeypatch.setattr(ops.NetworkProgram, "_launch", lambda network, build, program: program.zero_())

    def make(network, program, k):
        assert network.program is None and not hasattr(program, "_dl_tables")
        network.counted = 4
        made.append(torch.tensor(k))
        return made[-1]
    monkeypatch.setattr(ops.NetworkProgram, "_make_table", make)
    network.program = None
    network.build()
    assert {k: int(table) for k, table in network.program._dl_tables.items()} == {2: 2}


@pytest.fixture
def programs(cuda, monkeypatch):
    """Steps of NetworkProgram.build in place of launches; `left`: of 100 neurons, what is left as gates."""
    made = []
    library = type("Library", (), {"left": 0, "dl_network_program_words": lambda s, sizes, n: 8, "dl_network_whole_words": lambda s, sizes, n: 8,
                                   "dl_network_fold": "fold", "dl_network_order": lambda *a: made.append("order") or 0,
                                   "dl_network_whole": "whole"})()
    library.made = made

    def launch(network, build, program):
        made.append(build)
        program.fill_(library.left * sum(network.sizes[1:]) // 100)._dl_stream = 7
    monkeypatch.setattr(ops.N, "lib", lambda: library)
    monkeypatch.setattr(ops.N, "on_device", lambda t: ops.N._ALREADY_THERE)
    monkeypatch.setattr(ops.N, "stream_of", lambda t: 7)
    monkeypatch.setattr(ops.NetworkProgram, "_launch", launch)
    monkeypatch.setattr(ops.NetworkProgram, "_make_table", lambda network, program, k: made.append("table"))
    return library


def _unbuilt(rows):
    network = ops.NetworkProgram.__new__(ops.NetworkProgram)
    network.sizes, network.layers, network.program = (8, rows, rows), [(None, None, torch.zeros(8))] * 2, None
    return network


@pytest.mark.parametrize("rows,samples,folds", [(10240, 78644, True), (10240, 78643, False), (8000, 32768, False), (10241, 64, True)])
def test_small_passes_over_narrow_networks_do_not_fold(programs, rows, samples, folds):
    """Both sides of the lines; a network met by a small pass first is folded by the first one that is large enough."""
    network = _unbuilt(rows)
    network.samples = samples
    network.build()
    assert programs.made == (["fold", "order"] if folds else ["whole"])
    assert (network.limit is None) == folds and (network.program._dl_whole is None) == folds
    if not folds:
        assert not network.folds(network.limit - 1) and network.folds(network.limit)
        network.program._dl_tables[2] = None                   # two classes have been counted

        def words(samples):
            return torch.empty(8, samples // 64, dtype=torch.int64)
        assert network.serves(words(64 * 100), 2) and not network.serves(words(network.limit + 1024), 2)
        network.samples = network.limit
        network.build()
        assert programs.made == ["whole", "fold", "order"] and network.limit is None and network.program._dl_needs == (0, 0)


@pytest.mark.parametrize("small_first", [False, True])
@pytest.mark.parametrize("left,steps", [(74, ["fold", "order", "table"]), (75, ["fold", "whole"]), (100, ["fold", "whole"])])
def test_networks_that_do_not_fold_have_one_program(programs, left, steps, small_first):
    """How many gates are left is known before the rest of the folded program is made, and of what was made for it nothing stays."""
    programs.left = left
    network = _unbuilt(1000)
    network.counted = 2
    if small_first:
        network.samples = 64
        network.build()
        assert programs.made == ["whole"]
        del programs.made[:]
        steps = [step for step in steps if step != "whole"]     # which is there
    network.samples = 1 << 30
    network.build()
    assert programs.made == steps and network.limit is None
    kept = network.program
    assert (kept._dl_whole is not None) == (left >= 75) and (left < 75 or kept.untyped_storage().nbytes() == 16)


def test_uses_that_take_turns_build_each_program_once(cuda, argmax, monkeypatch):
    """The same layers counted in few classes (one kernel), in many (folded layers) and read as rows (one kernel)."""
    built, ran = [], []

    def build(network):
        built.append(type(network))
        network.program, network.pays, network.rows = torch.zeros(1), True, 8
        network.program._dl_tables = {network.counted: None}
    monkeypatch.setattr(ops, "_index", lambda t, name, n=None: None)
    monkeypatch.setattr(ops.N, "on_device", lambda t: ops.N._ALREADY_THERE)
    monkeypatch.setattr(ops.N, "stream_of", lambda t: 7)
    for kind in (ops.NetworkProgram, ops.FoldedLayers):
        monkeypatch.setattr(kind, "build", build)
    monkeypatch.setattr(ops, "eval_network_applicable", lambda x, sizes, batch, k: k < 4)
    monkeypatch.setattr(ops, "eval_folded_applicable", lambda x, sizes: True)
    monkeypatch.setattr(ops, "eval_folded_counts_applicable", lambda x, sizes, rows, k: True)
    monkeypatch.setattr(ops, "eval_groupbitsum_parts_applicable", lambda x, n_out, k: False)
    monkeypatch.setattr(ops, "eval_groupbitsum_applicable", lambda x, n_out, k: False)
    monkeypatch.setattr(ops, "groupbitsum", lambda x, pad_len, k, padded: "counts")
    monkeypatch.setattr(ops, "eval_packed", lambda x, a, b, gate: ran.append("layer") or x)
    monkeypatch.setattr(ops, "eval_network", lambda x, network, batch, k=None: ran.append("one kernel") or (x if k is None else "counts"))
    monkeypatch.setattr(ops, "eval_folded", lambda x, network, batch, k=None: ran.append("folded") or (x if k is None else "counts"))
    layers = [_layer(), _layer()]

    def use(k):
        del ran[:]
        packed = D.PackBitsTensor.from_packed(torch.ones(8, 2, dtype=torch.int64), 0)
        for layer in layers:
            packed._push_layer(layer)
        assert packed.t is not None if k is None else packed.group_sum(k) == "counts"
        return list(ran)
    uses = (2, 8, None)
    for k in uses:
        assert use(k) in (["layer"] * 2, ["one kernel"])
    for _ in range(3):
        assert [use(k) for k in uses] == [["one kernel"], ["folded"], ["one kernel"]]
    assert sorted(kind.__name__ for kind in built) == ["FoldedLayers", "NetworkProgram"]
    with torch.no_grad():
        layers[0].weights.add_(1.0)
    use(8)
    assert layers[1]._network is None and layers[1]._folded_network is not None     # nothing of other gates stays
    layers[1].train()
    assert layers[1]._folded_network is None and not {"_network", "_folded_network"} & set(layers[1].__getstate__())


@pytest.mark.parametrize("rows,k,words,together", [
    (20000, 5000, 2048, False), (20000, 2500, 64, True), (20000, 3001, 64, False), (20000, 3000, 64, True), (20000, 1250, 192, False),
    (20000, 1000, 192, True), (20000, 400, 2048, True), (47 * 400, 400, 512, False), (48 * 400, 400, 512, True), (3, 1, 1 << 12, True)])
def test_which_classes_are_counted_along_with_the_last_layer(monkeypatch, rows, k, words, together):
    """Both sides of the lines from which on a CTA per class and piece of the rows takes longer than rows and counts one after the other."""
    monkeypatch.setattr(ops, "eval_folded_counts_applicable", lambda x, sizes, rows, k: True)
    packed = D.PackBitsTensor.from_packed(torch.ones(8, words, dtype=torch.int64), 0)
    assert bool(packed._folded_counts((8, 9, rows), 9, k)) == together


@pytest.mark.parametrize("width,batch,training,evaluating", [
    (11999, 4096, False, False), (12000, 164, False, False), (12000, 168, True, True), (16000, 124, False, False), (16000, 128, True, True),
    (64000, 33, False, False), (64000, 64, False, False), (12000, 1024, True, True), (12000, 1028, True, False), (15999, 4096, True, False),
    (16000, 1028, True, True), (12000, 1027, True, True), (128000, 16, False, False), (128000, 17, True, True), (128000, 20, False, True),
    (128000, 28, True, True), (75776, 32, True, True), (75777, 32, False, True), (111999, 32, False, True), (112000, 32, True, True),
    (95999, 96, False, True), (96000, 68, True, True), (95999, 67, True, True), (40000, 100, True, True), (18944, 128, True, True),
    (18945, 128, False, True), (27999, 100, False, True), (28000, 128, True, True), (22499, 192, False, True), (22500, 192, True, True),
    (22499, 196, True, True), (20000, 129, True, True)])
def test_which_layers_take_the_walk(cuda, walks, width, batch, training, evaluating):
    """Both sides of every line at which the faster kernels change (a layer of few neurons stands in for one of many)."""
    layer = _layer()
    layer.out_dim = width
    assert (layer.train()._walk_for(batch) is not None) == training
    layer._walk = None
    layer.eval()
    assert [layer._walk_for(batch) is not None for _ in range(2)] == [False, evaluating]
