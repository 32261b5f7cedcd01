"""PackBitsTensor: a batch of boolean feature vectors packed along the batch dimension.

Drop-in for the reference class (difflogic/packbitstensor.py:6-41): `.t` is the packed tensor
`[features, ceil(batch / bit_count)]` of dtype int{bit_count}, `.pad_len` the number of unused
high bits in the last word, sample s being bit s % bit_count (LSB first) of word s // bit_count.

Rows are kept padded to whole units of 16 bytes while layers are applied, so that a batch of any size is moved 16 bytes
at a time by the kernels for long rows; `.t` shows the words of the batch only.

Evaluation is lazy.  A LogicLayer in eval mode does not compute at once; it appends itself to the
tensor's list of pending layers.  Layers of up to 16384 rows run in ONE kernel that keeps the activations
in shared memory (ops.eval_network): `group_sum(k)` -- what GroupSum calls -- gets the class counts from it,
reading `.t` the last layer's rows.  That kernel works from a program of the network, which mostly takes longer
to build than one batch takes without it; a network's first pass, and the first after its gates or connections
have changed, then runs one kernel per layer.  So do wider layers, exactly as the reference does, and
`group_sum(k)` then hands the last layer together with the bit-sum to one kernel that never stores the
layer's output (ops.eval_groupbitsum) when the sizes are in that kernel's range.  From the second pass on the wider
networks, too, run folded (ops.eval_folded): over the gates that are left when neurons that hand on a row or a constant,
and rows that nothing reads, are taken out.  The counts are
identical either way; the in-place semantics of the reference (the layer returns the same object, `.t`
then holds the layer's output) are kept.
"""
import os

import numpy as np
import torch

from . import ops


# Module switch, read from the environment once at import (set the attribute to change it afterwards).
FUSED_LAST_LAYER = os.environ.get("DL_FUSED_LAST_LAYER", "1") != "0"   # last layer + bit-sum in one kernel


# A network's first pass builds its program when the batch is as large, or no layer wider and the program that of all neurons.  First
# pass with the program / by single layers, us, host and build included, folded: 784 -> 4 x 8000: 2^13 246 / 161, 2^17 310 / 281, 2^18 366 /
# 428; 784 -> 5 x 16000: 2^15 312 / 224, 2^17 452 / 530; 784 -> 12 x 12000: 2^13 471 / 293, 2^16 520 / 575, 2^18 777 / 1753.  All neurons: 784 ->
# 2 x 2000: 2^10 samples 101 / 113, 2^17 111 / 118; 256 -> 12 x 4000: 2^13 267 / 261, 2^16 306 / 269.
PROGRAM_AT_ONCE_ROWS = 2000
PROGRAM_AT_ONCE_SAMPLES = 1 << 18

# Wider networks are folded in the first pass when their hidden rows take up this much memory.  The same figures: 784 -> 2 x 20000: 2^17
# samples (330 MB) 305 / 257; 9216 -> 4 x 128000: 10000 (490 MB) 369 / 363, 2^15 601 / 797; 256 -> 12 x 64000: 1000 (90 MB) 478 / 353, 10000
# (890 MB) 481 / 554, 2^17 1511 / 4509.
FOLD_AT_ONCE_BYTES = 5 << 27

# Classes of fewer neurons of a folded network than this are counted from the last layer's rows, unless (class, 512 bytes of a row) are at
# most so many: counting along with the layer takes a CTA for each and its 1.2 us for every CTA, however few neurons it has.  Whole passes
# of 784 -> 3 x 20000, us, counts with the layer / rows first, in classes of 4, 8, 16, 32, 50, 80 neurons: 2^17 samples 5591 / 3716,
# 2886 / 2119, 1537 / 1100, 818 / 720, 546 / 592, 393 / 488; 2^15 (8 pieces) 1408 / 925, 733 / 529, 396 / 283, 227 / 186, 165 / 154, 121 /
# 146; 10000 (3) 471 / 316, 253 / 193, 145 / 116, 89 / 98, 69 / 89, 55 / 84; 1000 (1) 96 / 76, 59 / 76, 52 / 75, 51 / 75.
FOLDED_COUNTS_NEURONS = 48
FOLDED_COUNTS_CTAS = 3000


class PackBitsTensor:
    def __init__(self, t: torch.BoolTensor, bit_count=32, device='cuda'):
        assert len(t.shape) == 2, t.shape

        self.bit_count = bit_count
        self.device = device
        self._pending = []

        if device == 'cuda' or (isinstance(device, (str, torch.device)) and torch.device(device).type == 'cuda'):
            t = t.to(device)
            if t.dtype != torch.bool:
                t = t != 0
            # transpose and pack in one kernel, straight from the batch-major matrix
            self._t, self.pad_len = ops.packbits_batch_major(t.contiguous(), self.bit_count, padded=True)
            self._words = -(-t.shape[0] // self.bit_count)
        else:
            raise NotImplementedError(device)

    @classmethod
    def from_packed(cls, words, pad_len, device='cuda'):
        """Wraps words that are already packed (e.g. a batch shard that was packed elsewhere)."""
        self = cls.__new__(cls)
        self.bit_count = ops.bits_of(words)
        self.device = device
        self._t = words
        self._words = words.shape[1]
        self._pending = []
        self.pad_len = int(pad_len)
        return self

    @classmethod
    def from_uint8_thresholds(cls, t, thresholds=(63, 127, 191), bit_count=64, device='cuda'):
        """Thermometer-encodes uint8 features (e.g. images `[batch, C, H, W]`) and packs them in one kernel.
        Feature `i * n + f` of the result is `t[:, f] > thresholds[i]` with f running over the flattened trailing
        dimensions -- the layout of `torch.cat([x > (i+1)/4 ...], dim=1)` followed by Flatten on `x = t / 255`."""
        t = t.to(device).reshape(t.shape[0], -1).contiguous()
        words, pad_len = ops.threshold_packbits_batch_major(t, thresholds, bit_count, padded=True)
        self = cls.from_packed(words, pad_len, device=device)
        self._words = -(-t.shape[0] // bit_count)
        return self

    # -- lazy layer application ------------------------------------------------------------------

    @property
    def t(self):
        """The packed tensor after every layer applied so far (pending layers run now)."""
        self._materialize()
        if self._t.shape[1] != self._words:
            self._t = self._t[:, :self._words].contiguous()
        return self._t

    @t.setter
    def t(self, value):
        self._pending = []
        self._t = value
        self._words = value.shape[1]

    def _push_layer(self, layer):
        """Called by LogicLayer.forward_cuda_eval: remember the layer (its connections and current arg-max gates)."""
        rows = self._pending[-1][0].out_dim if self._pending else self._t.shape[0]
        assert rows == layer.in_dim, ((rows,), layer.in_dim)
        self._pending.append((layer, layer._gates()))

    def _capturing(self):
        """Whether the pending layers, which are about to run, are being captured in a CUDA graph; their gates, from whenever they
        were applied, then stay with the layers."""
        if not torch.cuda.is_current_stream_capturing():
            return False
        for layer, gate in self._pending:
            layer._keep_for_graphs(gate)
        return True

    def _network(self, batch, k, counts=True):
        """The pending layers as a program for the one-kernel evaluation, None when that kernel does not take them, False when it
        is not their turn yet: where building the program takes longer than it saves one batch (PROGRAM_AT_ONCE_SAMPLES, _ROWS and
        FOLD_AT_ONCE_BYTES draw the line), it is built when the same gates and connections are met a second time.  It stays with the last layer until a layer's gates or connections
        are others, one of each kind: which one a pass takes goes by its classes and the alignment of its rows, too.  Not while a CUDA
        graph is being captured: the graph would outlive a program that a change of the weights replaces."""
        layers = [layer.indices + (gate,) for layer, gate in self._pending]
        last = self._pending[-1][0]
        kept = [last._network, last._folded_network]
        for i, network in enumerate(kept):
            if network is not None:
                if not (network.sizes[0] == self._t.shape[0] and network.matches(layers)):
                    kept[i] = None
                elif network.serves(self._t, k):
                    return network
                elif network.layer_by_layer:
                    return False
        any_kept = kept[0] or kept[1]
        sizes = any_kept.sizes if any_kept is not None else ops.network_sizes(self._t.shape[0], layers)
        narrow = max(sizes) <= ops.ONE_KERNEL_ROWS
        folded = not (narrow and ops.eval_network_applicable(self._t, sizes, batch, k))
        if folded and not ops.eval_folded_applicable(self._t, sizes):
            return None
        if folded and narrow and k > 1 and ops.eval_network_applicable(self._t, sizes, batch, 1) and not self._folded_counts(sizes, sum(sizes), k):
            return None                     # the classes are too many for the one kernel, not the layers
        network, samples = kept[folded], self._t.shape[1] * self.bit_count
        if network is None:
            device = self._t.get_device()
            counters = [ops.versions(a, b) for a, b, _ in layers]
            if None in counters or any(t.get_device() != device for layer in layers for t in layer):
                return None
            network = kept[folded] = (ops.FoldedLayers if folded else ops.NetworkProgram)(self._t.shape[0], layers, False, counters, sizes)
            last._network, last._folded_network = kept
            if folded:
                at_once = sum(sizes[1:-1]) * samples >= 8 * FOLD_AT_ONCE_BYTES
            else:
                at_once = samples >= PROGRAM_AT_ONCE_SAMPLES or (max(sizes[1:]) <= PROGRAM_AT_ONCE_ROWS and not network.folds(samples))
            if not at_once:
                return False
        if network.program is None or (network.limit is not None and samples >= network.limit):
            network.samples = samples
            if counts and (not folded or self._folded_counts(sizes, sum(sizes), k)):
                network.counted = k
            network.build()
        if folded and not network.pays:
            network.drop()
            # Three hidden layers or more that fit the one kernel run there all the same.  With gates that all need both inputs, us, one by
            # one / in one kernel: 784 -> 2 x 8000 -> 20000: 10000 samples 75 / 80, 2^17 207 / 245, 2^20 1456 / 1941; 4 x 8000: 102 / 87, 306 /
            # 278, 2195 / 2111; 12 x 8000: 202 / 109, 714 / 400, 5158 / 2976.  (With gates drawn evenly, folded / in one kernel: 4 x 8000: 62 /
            # 74, 166 / 284, 1152 / 2221.)
            hidden = sizes[:-1]
            return None if len(hidden) > 3 and ops.eval_network_applicable(self._t, ops.row_counts(hidden), batch, 1) else False
        return network

    def _run(self, network, batch, k=None):
        """The class counts of the pending layers, without k the last one's rows; None where there is no memory for the rows of
        a folded network (single layers need less)."""
        if not isinstance(network, ops.FoldedLayers):
            return ops.eval_network(self._t, network, batch, k)
        try:
            return ops.eval_folded(self._t, network, batch, k)
        except torch.cuda.OutOfMemoryError:
            return None

    def _materialize(self, in_one=True):
        if self._pending and self._capturing():
            in_one = False
        if in_one and len(self._pending) > 1:
            batch = self._t.shape[1] * self.bit_count
            network = self._network(batch, 1, counts=False)
            rows = self._run(network, batch) if network else None
            if rows is not None:
                self._t, self._pending = rows, []
                return
        pending, self._pending = self._pending, []
        for layer, gate in pending:
            a, b = layer.indices
            self._t = ops.eval_packed(self._t, a, b, gate)

    def group_sum(self, k):
        assert torch.device(self.device).type == 'cuda', self.device
        if not 0 <= self.pad_len < self.bit_count:
            raise RuntimeError('difflogic_b200: pad_len %d out of range' % self.pad_len)
        pad_len = self.pad_len + (self._t.shape[1] - self._words) * self.bit_count
        if self._pending and FUSED_LAST_LAYER:
            batch = self._t.shape[1] * self.bit_count - pad_len
            network = None if self._capturing() else self._network(batch, k)   # all layers are still pending
            if network and isinstance(network, ops.FoldedLayers) and not self._folded_counts(network.sizes, network.rows, k):
                self._materialize()
                return ops.groupbitsum(self._t, pad_len, k, padded=True)
            counts = self._run(network, batch, k) if network else None
            if counts is not None:
                return counts
            # all layers but the last run now; the last one is counted as it is computed, its output never stored
            (layer, gate) = self._pending.pop()
            self._materialize(in_one=network is None)
            self._pending.append((layer, gate))  # still pending: `.t` would run it as a kernel of its own
            how = self._counts_with_last_layer(layer.out_dim, k)
            if how:
                a, b = layer.indices
                return ops.eval_groupbitsum(self._t, a, b, gate, pad_len, k, parts=how == 'parts', padded=True)
        self._materialize()
        return ops.groupbitsum(self._t, pad_len, k, padded=True)

    def _folded_counts(self, sizes, rows, k):
        """Whether the classes of a folded network are counted along with its last layer."""
        pieces = -(-self._t.shape[1] * self._t.element_size() // 512)
        if k > 0 and sizes[len(sizes) - 1] < FOLDED_COUNTS_NEURONS * k and k * pieces > FOLDED_COUNTS_CTAS:
            return False
        return ops.eval_folded_counts_applicable(self._t, sizes, rows, k) or self._counts_with_last_layer(sizes[len(sizes) - 1], k)

    def _counts_with_last_layer(self, n_out, k):
        """Whether one kernel takes a last layer of n_out neurons together with the class counts: 'parts', 'whole' or None."""
        if ops.eval_groupbitsum_parts_applicable(self._t, n_out, k):
            return 'parts'
        return 'whole' if ops.eval_groupbitsum_applicable(self._t, n_out, k) else None

    def flatten(self, start_dim=0, end_dim=-1, **kwargs):
        """Returns the object itself so that torch.nn.Flatten passes it through; arguments are ignored."""
        return self

    def _row_repr(self, row):
        def word(v):
            return np.binary_repr(int(v), width=self.bit_count)[::-1]
        row = row.tolist()
        if len(row) <= 4:
            return ' '.join(word(v) for v in row)
        return '{} ... {}'.format(' '.join(word(v) for v in row[:3]), word(row[-1]))

    def __repr__(self):
        return '\n'.join(self._row_repr(row) for row in self.t.cpu())
