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
layer's output (ops.eval_groupbitsum) when the sizes are in that kernel's range.  The counts are
identical either way; the in-place semantics of the reference (the layer returns the same object, `.t`
then holds the layer's output) are kept.
"""
import os

import numpy as np
import torch

from . import ops


# Module switch, read from the environment once at import (set the attribute to change it afterwards).
FUSED_LAST_LAYER = os.environ.get("DL_FUSED_LAST_LAYER", "1") != "0"   # last layer + bit-sum in one kernel


# A network's first pass builds its program when no layer is wider, or the batch as large.  First pass with the program / by single
# layers, us, host and build included: 784 -> 2 x 2000: 2^10 samples 101 / 113, 2^17 111 / 118; 256 -> 12 x 4000: 2^13 267 / 261, 2^16 306 /
# 269; 784 -> 4 x 8000: 2^13 162 / 147, 2^17 256 / 267, 2^18 361 / 422; 784 -> 5 x 16000: 2^13 311 / 189, 2^17 573 / 532, 2^18 848 / 904;
# 784 -> 12 x 12000: 2^13 520 / 277, 2^18 1384 / 1722.
PROGRAM_AT_ONCE_ROWS = 2000
PROGRAM_AT_ONCE_SAMPLES = 1 << 18


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

    def _network(self, batch, k):
        """The pending layers as a program for the one-kernel evaluation, None when that kernel does not take them, False when it
        is not their turn yet: where building the program takes longer than it saves one batch (PROGRAM_AT_ONCE_ROWS), it is built
        when the same gates and connections are met a second time.  It stays with the last layer until a layer's gates or connections are others.  Not while a CUDA
        graph is being captured: the graph would outlive a program that a change of the weights replaces."""
        layers = [layer.indices + (gate,) for layer, gate in self._pending]
        last = self._pending[-1][0]
        network = last._network
        if network is not None and not (network.sizes[0] == self._t.shape[0] and network.matches(layers)):
            network = None
        sizes = network.sizes if network is not None else ops.network_sizes(self._t.shape[0], layers)
        if not ops.eval_network_applicable(self._t, sizes, batch, k):
            return None
        if network is None:
            if any(t.device != self._t.device for layer in layers for t in layer) or any(ops.versions(a, b) is None for a, b, _ in layers):
                return None
            network = last._network = ops.NetworkProgram(self._t.shape[0], layers, build=False)
            if max(network.sizes[1:]) > PROGRAM_AT_ONCE_ROWS and self._t.shape[1] * self.bit_count < PROGRAM_AT_ONCE_SAMPLES:
                return False
        if network.program is None:
            network.build()
        return network

    def _materialize(self, in_one=True):
        if self._pending and self._capturing():
            in_one = False
        if in_one and len(self._pending) > 1:
            batch = self._t.shape[1] * self.bit_count
            network = self._network(batch, 1)
            if network:
                self._t, self._pending = ops.eval_network(self._t, network, batch), []
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
            network = None if self._capturing() else self._network(batch, k)
            if network:
                return ops.eval_network(self._t, network, batch, k)   # all layers are still pending
            # all layers but the last run now; the last one is counted as it is computed, its output never stored
            (layer, gate) = self._pending.pop()
            self._materialize(in_one=network is None)
            self._pending.append((layer, gate))  # still pending: `.t` would run it as a kernel of its own
            parts = ops.eval_groupbitsum_parts_applicable(self._t, layer.out_dim, k)
            if parts or ops.eval_groupbitsum_applicable(self._t, layer.out_dim, k):
                a, b = layer.indices
                return ops.eval_groupbitsum(self._t, a, b, gate, pad_len, k, parts=parts, padded=True)
        self._materialize()
        return ops.groupbitsum(self._t, pad_len, k, padded=True)

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
