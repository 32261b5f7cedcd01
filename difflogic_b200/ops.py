"""Tensor-level operators over the C ABI (include/difflogic_b200.h).

Each function checks its tensors, lets torch allocate the output on the inputs' device and
launches the kernel on torch's current stream.  Nothing here computes on the CPU; a missing
library raises (see _native.lib()).

Layouts: float activations are feature-major `[features, batch]` contiguous; packed
activations are `[features, words]`; indices are int64, as LogicLayer stores them.
"""
import collections

import torch

from . import _native as N
from ._native import W_ARGMAX, W_LOGITS, W_PROBS  # noqa: F401  (re-exported)

_BITS_TO_DTYPE = {8: torch.int8, 16: torch.int16, 32: torch.int32, 64: torch.int64}
_DTYPE_TO_BITS = {v: k for k, v in _BITS_TO_DTYPE.items()}
_DTYPE_TO_BITS[torch.uint8] = 8


def _need(cond, msg):
    if not cond:
        raise RuntimeError("difflogic_b200: " + msg)


def _f32_matrix(t, name):
    if t.is_cuda and t.dtype is torch.float32 and t.dim() == 2 and t.is_contiguous():
        return
    N.require_cuda(t)
    _need(t.dtype == torch.float32, "%s must be float32, got %s (the CUDA path computes in fp32)" % (name, t.dtype))
    _need(t.dim() == 2 and t.is_contiguous(), "%s must be a contiguous 2-D tensor" % name)


def _index(t, name, n=None):
    if t.is_cuda and t.dtype is torch.int64 and t.dim() == 1 and t.is_contiguous() and (n is None or t.numel() == n):
        return
    N.require_cuda(t)
    _need(t.dtype == torch.int64 and t.dim() == 1 and t.is_contiguous(), "%s must be a contiguous int64 vector" % name)
    if n is not None:
        _need(t.numel() == n, "%s has %d entries, expected %d" % (name, t.numel(), n))


# ------------------------------------------------------------------------------------------------
# training
# ------------------------------------------------------------------------------------------------

def logic_forward(x, a, b, w, w_mode=W_LOGITS, want_coef=False, overlap=False):
    """y[j,:] = sum_i p[j,i] gate_i(x[a_j,:], x[b_j,:]);  returns (y [n_out,batch], coef or None).

    overlap=True lets the kernel read `a`, `b` while the previous kernel in the stream is still running; pass
    it only when those index tensors were complete before that kernel was launched (see DL_LAUNCH_OVERLAP_SETUP)."""
    _f32_matrix(x, "x")
    _f32_matrix(w, "w")
    n_in, batch = x.shape
    n_out = w.shape[0]
    _need(w.shape[1] == 16, "w must be [n_out, 16]")
    _index(a, "a", n_out)
    _index(b, "b", n_out)
    y = x.new_empty((n_out, batch))
    coef = x.new_empty((n_out, 4)) if want_coef else None
    with N.on_device(x):
        N.check(N.lib().dl_forward_f32(x.data_ptr(), a.data_ptr(), b.data_ptr(), w.data_ptr(), w_mode, y.data_ptr(),
                                       N.ptr(coef), n_in, n_out, batch, int(overlap), N.stream_of(x)))
    return y, coef


def logic_coefs(w, w_mode=W_LOGITS):
    _f32_matrix(w, "w")
    _need(w.shape[1] == 16, "w must be [n_out, 16]")
    coef = torch.empty((w.shape[0], 4), dtype=torch.float32, device=w.device)
    with N.on_device(w):
        N.check(N.lib().dl_coefs_f32(w.data_ptr(), w_mode, coef.data_ptr(), w.shape[0], N.stream_of(w)))
    return coef


def transpose(x):
    """[rows, cols] float32 -> its transpose as a new contiguous tensor (dl_transpose_f32)."""
    _f32_matrix(x, "x")
    y = x.new_empty((x.shape[1], x.shape[0]))
    with N.on_device(x):
        N.check(N.lib().dl_transpose_f32(x.data_ptr(), y.data_ptr(), x.shape[0], x.shape[1], N.stream_of(x)))
    return y


def logic_backward_w(x, a, b, grad_y, w=None, w_mode=W_PROBS, out=None, overlap=False, rows_per_class=1):
    """[n_out,16] gradient: w_mode=W_PROBS w.r.t. the mixing weights, W_LOGITS w.r.t. the raw
    parameters `w` (softmax backward applied in the kernel).  rows_per_class > 1: grad_y holds one row per class of
    that many consecutive outputs (the gradient that comes back through a GroupSum), [n_out / rows_per_class, batch]."""
    _f32_matrix(x, "x")
    _f32_matrix(grad_y, "grad_y")
    n_in, batch = x.shape
    rows_per_class = int(rows_per_class)
    _need(rows_per_class >= 1, "rows_per_class must be positive")
    n_out = grad_y.shape[0] * rows_per_class
    _need(grad_y.shape[1] == batch, "grad_y and x disagree on the batch size")
    _index(a, "a", n_out)
    _index(b, "b", n_out)
    if w_mode == W_LOGITS:
        _need(w is not None, "W_LOGITS needs the raw weights")
        _f32_matrix(w, "w")
        _need(tuple(w.shape) == (n_out, 16), "w must be [n_out, 16]")
    if out is None:
        out = x.new_empty((n_out, 16))
    else:
        _f32_matrix(out, "out")
        _need(tuple(out.shape) == (n_out, 16), "out must be [n_out, 16]")
    with N.on_device(x):
        if rows_per_class == 1:
            N.check(N.lib().dl_backward_w_f32(x.data_ptr(), a.data_ptr(), b.data_ptr(), grad_y.data_ptr(), N.ptr(w), w_mode,
                                              out.data_ptr(), n_in, n_out, batch, int(overlap), N.stream_of(x)))
        else:
            N.check(N.lib().dl_backward_w_classes_f32(x.data_ptr(), a.data_ptr(), b.data_ptr(), grad_y.data_ptr(), N.ptr(w), w_mode,
                                                      out.data_ptr(), n_in, n_out, batch, rows_per_class, int(overlap),
                                                      N.stream_of(x)))
    return out


def logic_backward_w_adam(x, a, b, grad_y, w, exp_avg, exp_avg_sq, state, lr, beta1, beta2, eps, grad_scale=1.0, grad_out=None,
                          overlap=False, rows_per_class=1):
    """backward_w of a layer with the Adam step of its weights in the kernel's epilogue: `w` [n_out, 16] and its moment
    slices are updated in place; the gradient is stored only when `grad_out` is given.  `state`: two int32 on the device
    that belong to this layer, {steps done, 0}; the kernel advances the count."""
    _f32_matrix(x, "x")
    _f32_matrix(grad_y, "grad_y")
    _f32_matrix(w, "w")
    n_in, batch = x.shape
    rows_per_class = int(rows_per_class)
    n_out = grad_y.shape[0] * rows_per_class
    _need(grad_y.shape[1] == batch, "grad_y and x disagree on the batch size")
    _need(tuple(w.shape) == (n_out, 16), "w must be [n_out, 16]")
    _index(a, "a", n_out)
    _index(b, "b", n_out)
    for t, name in ((exp_avg, "exp_avg"), (exp_avg_sq, "exp_avg_sq")):
        _need(t.is_cuda and t.dtype == torch.float32 and t.is_contiguous() and t.numel() >= n_out * 16 and t.device == x.device,
              "%s must be a contiguous float32 CUDA tensor of at least n_out * 16 elements" % name)
    _need(state.is_cuda and state.dtype == torch.int32 and state.numel() >= 2 and state.is_contiguous(),
          "state must be a contiguous int32 CUDA tensor of two elements")
    if grad_out is not None:
        _f32_matrix(grad_out, "grad_out")
        _need(tuple(grad_out.shape) == (n_out, 16), "grad_out must be [n_out, 16]")
    with N.on_device(x):
        N.check(N.lib().dl_backward_w_adam_f32(x.data_ptr(), a.data_ptr(), b.data_ptr(), grad_y.data_ptr(), w.data_ptr(),
                                               exp_avg.data_ptr(), exp_avg_sq.data_ptr(), N.ptr(grad_out), n_in, n_out, batch,
                                               rows_per_class, float(lr), float(beta1), float(beta2), float(eps), float(grad_scale),
                                               state.data_ptr(), int(overlap), N.stream_of(x)))
    return grad_out


def logic_backward_w_announce(x, a, b, grad_y, w, out, rows_per_class, flag_ptrs, rank, world, bucket, bucket_state, block_ticket,
                              kernel_count, kernels_in_bucket):
    """logic_backward_w (W_LOGITS) into `out` [n_out, 16] whose last block announces the gradients of exchange bucket
    `bucket` to the peers (dl_backward_w_announce_f32).  flag_ptrs: ctypes array of the ranks' flag words;
    bucket_state / block_ticket / kernel_count: int32 device tensors (see the header)."""
    _f32_matrix(x, "x")
    _f32_matrix(grad_y, "grad_y")
    _f32_matrix(w, "w")
    _f32_matrix(out, "out")
    n_in, batch = x.shape
    rows_per_class = int(rows_per_class)
    n_out = grad_y.shape[0] * rows_per_class
    _need(grad_y.shape[1] == batch, "grad_y and x disagree on the batch size")
    _need(tuple(w.shape) == (n_out, 16) and tuple(out.shape) == (n_out, 16), "w and out must be [n_out, 16]")
    _index(a, "a", n_out)
    _index(b, "b", n_out)
    for t in (bucket_state, block_ticket, kernel_count):
        _need(t.is_cuda and t.dtype == torch.int32 and t.numel() >= 1, "state words must be int32 CUDA tensors")
    with N.on_device(x):
        N.check(N.lib().dl_backward_w_announce_f32(x.data_ptr(), a.data_ptr(), b.data_ptr(), grad_y.data_ptr(), w.data_ptr(),
                                                   out.data_ptr(), n_in, n_out, batch, rows_per_class, flag_ptrs, rank, world, bucket,
                                                   bucket_state.data_ptr(), block_ticket.data_ptr(), kernel_count.data_ptr(),
                                                   int(kernels_in_bucket), N.LAUNCH_OVERLAP_SETUP, N.stream_of(x)))
    return out


def inverse_index(a, b, n_in):
    """The reference's inverse connection index (difflogic/difflogic.py:56-69) built with device
    ops: for every input row the consumer neurons in increasing order, a neuron whose two inputs
    are the same row listed twice.  Returns (start [n_in+1] int64, list [2*n_out] int64)."""
    keys = torch.stack([a, b], dim=1).reshape(-1)           # position 2*j + slot
    order = torch.argsort(keys, stable=True)
    counts = torch.bincount(keys, minlength=n_in)
    start = torch.zeros(n_in + 1, dtype=torch.int64, device=a.device)
    start[1:] = torch.cumsum(counts, 0)
    return start, (order // 2).contiguous()


def build_backward_plan(a, b, start, lst):
    n_out = a.numel()
    n_in = start.numel() - 1
    _index(a, "a")
    _index(b, "b", n_out)
    _index(start, "start")
    _index(lst, "list", 2 * n_out)
    plan = torch.empty((2 * n_out, 2), dtype=torch.int32, device=a.device)
    with N.on_device(a):
        N.check(N.lib().dl_build_backward_plan(a.data_ptr(), b.data_ptr(), start.data_ptr(), lst.data_ptr(),
                                               plan.data_ptr(), n_in, n_out, N.stream_of(a)))
    return plan


def versions(*tensors):
    """Version counters of tensors that something is derived from and kept, or None when one of them has none (tensors made in
    inference mode): in-place writes to them go unnoticed, and nothing may be kept."""
    return None if any(t.is_inference() for t in tensors) else tuple(t._version for t in tensors)


class Walk(collections.namedtuple("Walk", "entries complete n_in n_out")):
    """Walk of a layer's connection graph: entries int32 [n, 2] on the device; complete: it gives grad_x; the layer's rows."""
    __slots__ = ()


def build_walk(a, b, n_in):
    """Walk of a layer's connection graph for logic_forward_walk / logic_backward_walk, or None for sizes or indices it does
    not take.  Built on the host (dl_build_walk)."""
    import ctypes
    n_out = a.numel()
    _index(a, "a")
    _index(b, "b", n_out)
    if n_out == 0 or n_in == 0:
        return None
    ah, bh = a.cpu().contiguous(), b.cpu().contiguous()
    out = torch.empty((N.lib().dl_walk_capacity(int(n_in), n_out), 2), dtype=torch.int32)
    entries, complete = ctypes.c_int64(), ctypes.c_int()
    if N.lib().dl_build_walk(ah.data_ptr(), bh.data_ptr(), int(n_in), n_out, out.data_ptr(), ctypes.addressof(entries),
                             ctypes.addressof(complete)) != N.DL_OK:
        return None
    return Walk(out[:entries.value].to(a.device), bool(complete.value), int(n_in), n_out)


def _check_walk(walk, n_in, n_out):
    """The walk's entries are row numbers: of x and of everything that has a row per neuron."""
    _need(n_in == walk.n_in, "x has %d rows, the walk's layer reads %d" % (n_in, walk.n_in))
    _need(n_out == walk.n_out, "w has %d rows, expected %d" % (n_out, walk.n_out))


def logic_forward_walk(x, w, walk, w_mode=W_LOGITS, want_coef=False, overlap=False):
    """logic_forward along the layer's walk (build_walk): same result, one row load per neuron."""
    _f32_matrix(x, "x")
    _f32_matrix(w, "w")
    n_in, batch = x.shape
    n_out = w.shape[0]
    _need(w.shape[1] == 16, "w must be [n_out, 16]")
    _check_walk(walk, n_in, n_out)
    y = x.new_empty((n_out, batch))
    coef = x.new_empty((n_out, 4)) if want_coef else None
    with N.on_device(x):
        N.check(N.lib().dl_forward_walk_f32(x.data_ptr(), w.data_ptr(), w_mode, y.data_ptr(), N.ptr(coef), walk[0].data_ptr(),
                                            walk[0].shape[0], n_in, n_out, batch, int(overlap), N.stream_of(x)))
    return y, coef


def logic_backward_walk(x, grad_y, coef, w, walk, grad_scale=1.0, want_grad_x=True, grad_out=None, adam=None, overlap=False,
                        rows_per_class=1):
    """backward_w and backward_x of a layer in one pass along its walk: (grad_x or None, grad_w or None).  adam: what
    FlatAdam.backward_args gives; the weights are then updated in place and grad_w is stored only into grad_out."""
    _f32_matrix(x, "x")
    _f32_matrix(grad_y, "grad_y")
    _f32_matrix(coef, "coef")
    _f32_matrix(w, "w")
    n_in, batch = x.shape
    n_out = w.shape[0]
    rows_per_class = int(rows_per_class)
    _check_walk(walk, n_in, n_out)
    _need(tuple(grad_y.shape) == (n_out // max(rows_per_class, 1), batch), "grad_y does not fit x and w")
    _need(tuple(w.shape) == (n_out, 16) and tuple(coef.shape) == (n_out, 4), "w must be [n_out, 16] and coef [n_out, 4]")
    gx = torch.empty_like(x) if want_grad_x else None
    if adam is None and grad_out is None:
        grad_out = x.new_empty((n_out, 16))
    if grad_out is not None:
        _f32_matrix(grad_out, "grad_out")
        _need(tuple(grad_out.shape) == (n_out, 16), "grad_out must be [n_out, 16]")
    a = adam or {}
    with N.on_device(x):
        N.check(N.lib().dl_backward_walk_f32(x.data_ptr(), grad_y.data_ptr(), coef.data_ptr(), w.data_ptr(), N.ptr(grad_out), N.ptr(gx),
                                             float(grad_scale), walk[0].data_ptr(), walk[0].shape[0], int(walk[1]), n_in, n_out, batch,
                                             rows_per_class, N.ptr(a.get("exp_avg")), N.ptr(a.get("exp_avg_sq")), float(a.get("lr", 0.0)),
                                             float(a.get("beta1", 0.0)), float(a.get("beta2", 0.0)), float(a.get("eps", 0.0)),
                                             float(a.get("grad_scale", 1.0)), N.ptr(a.get("state")), int(overlap), N.stream_of(x)))
    return gx, grad_out


_VIOLATIONS = {1: "connection index outside [0, in_dim)", 2: "inverse-index offsets are not 0 = start[0] <= ... <= start[in_dim] = 2 * out_dim",
               3: "inverse-index entry outside [0, out_dim)", 4: "gather-plan entry out of range",
               5: "gather-plan entry does not match the connections"}


def logic_backward_w_push(x, a, b, grad_y, w, out, rows_per_class, grad_inbox_ptrs, rank, world, bucket_offset, bucket_count,
                          inbox_offset, inbox_stride, bucket_state):
    """logic_backward_w (W_LOGITS) into `out` [n_out, 16] that also pushes the gradients of the other ranks' slices of the
    exchange bucket into their inboxes as packets (dl_backward_w_push_f32).  grad_inbox_ptrs: ctypes array of the ranks'
    gradient inboxes; bucket_offset / bucket_count: floats in front of this layer inside the bucket / of the bucket."""
    _f32_matrix(x, "x")
    _f32_matrix(grad_y, "grad_y")
    _f32_matrix(w, "w")
    _f32_matrix(out, "out")
    n_in, batch = x.shape
    rows_per_class = int(rows_per_class)
    n_out = grad_y.shape[0] * rows_per_class
    _need(grad_y.shape[1] == batch, "grad_y and x disagree on the batch size")
    _need(tuple(w.shape) == (n_out, 16) and tuple(out.shape) == (n_out, 16), "w and out must be [n_out, 16]")
    _index(a, "a", n_out)
    _index(b, "b", n_out)
    with N.on_device(x):
        N.check(N.lib().dl_backward_w_push_f32(x.data_ptr(), a.data_ptr(), b.data_ptr(), grad_y.data_ptr(), w.data_ptr(), out.data_ptr(),
                                               n_in, n_out, batch, rows_per_class, grad_inbox_ptrs, int(rank), int(world),
                                               int(bucket_offset), int(bucket_count), int(inbox_offset), int(inbox_stride),
                                               bucket_state.data_ptr(), N.LAUNCH_OVERLAP_SETUP, N.stream_of(x)))
    return out


def check_connections(a, b, n_in, start=None, lst=None, plan=None):
    """Checks a layer's index tensors on the device (dl_check_connections) and raises ValueError with the first violation
    found.  Synchronises; meant for construction time and debugging, not for the hot path."""
    n_out = a.numel()
    _index(a, "a")
    _index(b, "b", n_out)
    if start is not None:
        _index(start, "start", n_in + 1)
    if lst is not None:
        _index(lst, "list", 2 * n_out)
    if plan is not None:
        _need(plan.is_cuda and plan.dtype == torch.int32 and plan.is_contiguous() and tuple(plan.shape) == (2 * n_out, 2),
              "plan must be a contiguous int32 [2*n_out, 2] tensor")
    report = torch.zeros(4, dtype=torch.int64, device=a.device)
    with N.on_device(a):
        N.check(N.lib().dl_check_connections(a.data_ptr(), b.data_ptr(), N.ptr(start), N.ptr(lst), N.ptr(plan), int(n_in), n_out,
                                             report.data_ptr(), N.stream_of(a)))
    code, where, value, limit = report.tolist()
    if code != 0:
        raise ValueError("difflogic_b200: %s (position %d, value %d, limit %d)" % (_VIOLATIONS.get(code, "violation %d" % code),
                                                                                 where, value, limit))


def logic_backward_x(x, coef, grad_y, start, plan, grad_scale=1.0, overlap=False, rows_per_class=1):
    """Gradient w.r.t. the layer's input.  rows_per_class > 1: grad_y holds one row per class (see logic_backward_w)."""
    _f32_matrix(x, "x")
    _f32_matrix(grad_y, "grad_y")
    _f32_matrix(coef, "coef")
    n_in, batch = x.shape
    rows_per_class = int(rows_per_class)
    _need(rows_per_class >= 1, "rows_per_class must be positive")
    n_out = grad_y.shape[0] * rows_per_class
    _need(grad_y.shape[1] == batch, "grad_y and x disagree on the batch size")
    _need(tuple(coef.shape) == (n_out, 4), "coef must be [n_out, 4]")
    _index(start, "start", n_in + 1)
    N.require_cuda(plan)
    _need(plan.dtype == torch.int32 and plan.is_contiguous() and tuple(plan.shape) == (2 * n_out, 2),
          "plan must be a contiguous int32 [2*n_out, 2] tensor")
    gx = torch.empty_like(x)
    with N.on_device(x):
        if rows_per_class == 1:
            N.check(N.lib().dl_backward_x_f32(x.data_ptr(), coef.data_ptr(), grad_y.data_ptr(), start.data_ptr(),
                                              plan.data_ptr(), float(grad_scale), gx.data_ptr(), n_in, n_out, batch,
                                              int(overlap), N.stream_of(x)))
        else:
            N.check(N.lib().dl_backward_x_classes_f32(x.data_ptr(), coef.data_ptr(), grad_y.data_ptr(), start.data_ptr(),
                                                      plan.data_ptr(), float(grad_scale), gx.data_ptr(), n_in, n_out, batch,
                                                      rows_per_class, int(overlap), N.stream_of(x)))
    return gx


# ------------------------------------------------------------------------------------------------
# packed-bit inference
# ------------------------------------------------------------------------------------------------

def bits_of(t):
    _need(t.dtype in _DTYPE_TO_BITS, "packed tensor must be int8/int16/int32/int64, got %s" % t.dtype)
    return _DTYPE_TO_BITS[t.dtype]


def argmax_gates(w):
    _f32_matrix(w, "w")
    _need(w.shape[1] == 16, "w must be [n_out, 16]")
    g = torch.empty((w.shape[0],), dtype=torch.uint8, device=w.device)
    with N.on_device(w):
        N.check(N.lib().dl_argmax_gate_u8(w.data_ptr(), g.data_ptr(), w.shape[0], N.stream_of(w)))
    return g


def eval_packed(x, a, b, gate, out=None):
    N.require_cuda(x, gate)
    _need(x.dim() == 2 and x.is_contiguous(), "x must be a contiguous 2-D tensor")
    bits = bits_of(x)
    n_in, words = x.shape
    n_out = gate.numel()
    _need(gate.dtype == torch.uint8 and gate.is_contiguous(), "gate must be a contiguous uint8 vector")
    _index(a, "a", n_out)
    _index(b, "b", n_out)
    if out is None:
        out = torch.empty((n_out, words), dtype=x.dtype, device=x.device)
    else:
        _need(out.dtype == x.dtype and tuple(out.shape) == (n_out, words) and out.is_contiguous() and out.is_cuda,
              "out must be a contiguous [n_out, words] tensor of x's dtype")
        _need(out.data_ptr() != x.data_ptr(), "eval_packed cannot run in place")
    with N.on_device(x):
        N.check(N.lib().dl_eval_packed(x.data_ptr(), a.data_ptr(), b.data_ptr(), gate.data_ptr(), out.data_ptr(),
                                       n_in, n_out, words, bits, N.stream_of(x)))
    return out


def _as_bool_bytes(t):
    N.require_cuda(t)
    _need(t.dim() == 2 and t.is_contiguous(), "t must be a contiguous 2-D tensor")
    _need(t.dtype in (torch.bool, torch.uint8), "t must be a bool tensor, got %s" % t.dtype)
    return t


def _check_bit_count(bit_count):
    if bit_count not in _BITS_TO_DTYPE:
        raise ValueError("`bit_count` has to be in { 8, 16, 32, 64 }")


def packbits(t, bit_count):
    """bool [n, batch] (feature-major) -> (words [n, ceil(batch/bit_count)], pad_len)."""
    _check_bit_count(bit_count)
    t = _as_bool_bytes(t)
    n, batch = t.shape
    words = -(-batch // bit_count)
    out = torch.empty((n, words), dtype=_BITS_TO_DTYPE[bit_count], device=t.device)
    with N.on_device(t):
        N.check(N.lib().dl_packbits(t.data_ptr(), out.data_ptr(), n, batch, bit_count, N.stream_of(t)))
    return out, (bit_count - batch % bit_count) % bit_count


ROW_UNIT_BITS = 128   # rows padded to units of 16 bytes: what the packed kernels move at a time


def packbits_batch_major(t, bit_count, padded=False):
    """bool [batch, n] (as the user holds it) -> (words [n, ceil(batch/bit_count)], pad_len).  padded: the rows are filled
    up with zero words to whole units of 16 bytes."""
    _check_bit_count(bit_count)
    t = _as_bool_bytes(t)
    batch, n = t.shape
    unit = ROW_UNIT_BITS if padded else bit_count
    out = torch.empty((n, -(-batch // unit) * (unit // bit_count)), dtype=_BITS_TO_DTYPE[bit_count], device=t.device)
    with N.on_device(t):
        N.check(N.lib().dl_packbits_batch_major(t.data_ptr(), out.data_ptr(), n, batch, unit, N.stream_of(t)))
    return out, (bit_count - batch % bit_count) % bit_count


def threshold_packbits_batch_major(t, thresholds, bit_count, padded=False):
    """uint8 [batch, n] -> (words [len(thresholds)*n, ceil(batch/bit_count)], pad_len); bit s of row i*n+f is
    t[s, f] > thresholds[i] (thermometer encoding and packing in one kernel).  padded: as in packbits_batch_major."""
    import ctypes
    _check_bit_count(bit_count)
    N.require_cuda(t)
    _need(t.dim() == 2 and t.is_contiguous() and t.dtype == torch.uint8, "t must be a contiguous 2-D uint8 tensor")
    thresholds = [int(v) for v in thresholds]
    _need(1 <= len(thresholds) <= 16 and all(0 <= v <= 255 for v in thresholds), "1..16 thresholds in 0..255")
    batch, n = t.shape
    unit = ROW_UNIT_BITS if padded else bit_count
    out = torch.empty((len(thresholds) * n, -(-batch // unit) * (unit // bit_count)), dtype=_BITS_TO_DTYPE[bit_count], device=t.device)
    arr = (ctypes.c_ubyte * len(thresholds))(*thresholds)
    with N.on_device(t):
        N.check(N.lib().dl_threshold_packbits_batch_major(t.data_ptr(), ctypes.addressof(arr), len(thresholds), out.data_ptr(),
                                                          n, batch, unit, N.stream_of(t)))
    return out, (bit_count - batch % bit_count) % bit_count


def _row_units(x, padded):
    """(units, bits per unit) of the rows of x for a count: its words, or units of 16 bytes (rows padded to those)."""
    bits = bits_of(x)
    words = x.shape[1]
    if padded and words * bits % ROW_UNIT_BITS == 0:
        return words * bits // ROW_UNIT_BITS, ROW_UNIT_BITS
    return words, bits


def groupbitsum(x, pad_len, k, padded=False):
    """words [n, W] -> int32 [W*bits - pad_len, k] class counts.  pad_len: samples of the last word that are left out; of the last
    16 bytes with `padded`."""
    N.require_cuda(x)
    _need(x.dim() == 2 and x.is_contiguous(), "x must be a contiguous 2-D tensor")
    words, bits = _row_units(x, padded)
    n = x.shape[0]
    k = int(k)
    if k <= 0 or n % k != 0:
        raise ValueError("in_dim (%d) has to be divisible by k (%d) but it is not" % (n, k))
    batch = words * bits - int(pad_len)
    _need(batch >= 0, "pad_len exceeds the packed batch")
    out = torch.empty((batch, k), dtype=torch.int32, device=x.device)
    with N.on_device(x):
        N.check(N.lib().dl_groupbitsum(x.data_ptr(), out.data_ptr(), n, words, int(pad_len), k, bits, N.stream_of(x)))
    return out


def eval_groupbitsum_applicable(x, n_out, k):
    """True when the fused last-layer + group bit-sum kernel takes a layer of n_out gates on packed words x."""
    if not (x.is_cuda and x.dim() == 2 and x.is_contiguous()):
        return False
    n_in, words = x.shape
    return N.lib().dl_eval_groupbitsum_applicable(x.data_ptr(), n_in, int(n_out), words, bits_of(x), int(k)) == 1


def eval_groupbitsum_parts_applicable(x, n_out, k):
    """The same for classes longer than that kernel's counters (eval_groupbitsum(..., parts=True))."""
    if not (x.is_cuda and x.dim() == 2 and x.is_contiguous()):
        return False
    n_in, words = x.shape
    return N.lib().dl_eval_groupbitsum_parts_applicable(x.data_ptr(), n_in, int(n_out), words, bits_of(x), int(k)) == 1


def eval_groupbitsum(x, a, b, gate, pad_len, k, parts=False, padded=False):
    """groupbitsum(eval_packed(x, a, b, gate), pad_len, k, padded) in one kernel; the layer's output is never stored.  parts:
    classes of more than 2040 gates, counted in parts."""
    N.require_cuda(x, a, b, gate)
    _need(x.dim() == 2 and x.is_contiguous(), "x must be a contiguous 2-D tensor")
    _need(a.dtype == torch.int64 and b.dtype == torch.int64 and gate.dtype == torch.uint8, "a, b int64 and gate uint8")
    _need(a.numel() == b.numel() == gate.numel(), "a, b and gate must have one entry per gate")
    words, bits = _row_units(x, padded)
    n_in = x.shape[0]
    n_out, k = a.numel(), int(k)
    if k <= 0 or n_out % k != 0:
        raise ValueError("in_dim (%d) has to be divisible by k (%d) but it is not" % (n_out, k))
    batch = words * bits - int(pad_len)
    _need(batch >= 0, "pad_len exceeds the packed batch")
    out = torch.empty((batch, k), dtype=torch.int32, device=x.device)
    with N.on_device(x):
        run = N.lib().dl_eval_groupbitsum_parts if parts else N.lib().dl_eval_groupbitsum
        N.check(run(x.data_ptr(), a.data_ptr(), b.data_ptr(), gate.data_ptr(), out.data_ptr(), n_in, n_out, words, int(pad_len), k, bits,
                    N.stream_of(x)))
    return out


# Layers of up to FOLD_ROWS rows are folded for passes of this many neurons x samples; smaller passes evaluate all neurons: that program is
# four launches for four layers, the folded one 26 and a table, and what its kernel saves does not show where the host takes longer than
# the GPU.  Second pass, with the build / pass among others, us, all neurons / folded: 784 -> 4 x 2000: 10000 samples 65 / 203, 42 / 41, 2^17
# 86 / 240, 56 / 56; 4 x 8000: 100 samples 176 / 208, 42 / 42 (the kernel 14.4 / 15.7), 2^15 200 / 217, 43 / 42, 2^16 (225) / 236, 75 / 48;
# 256 -> 12 x 4000: 10000 274 / 369, 60 / 59, 2^15 287 / 365, 61 / 61, 2^16 (318) / 379, 74 / 59.  Of wider layers the program of all neurons
# takes longer to build, one CTA per layer: 784 -> 5 x 16000, 100 samples (301) / 236, 10000 (322) / 240, 51 / 43.
FOLD_WORK = 3 << 29
FOLD_ROWS = 10240


class NetworkProgram:
    """What dl_eval_network needs of a network: its row counts and its program (dl_network_program), built from the layers'
    connections and arg-max gates.  `layers`: (a, b, gate) of every layer, in order; they are kept, so that `matches` can
    tell a network by its tensors.  build=False leaves the program to a later build()."""

    def __init__(self, n_in, layers, build=True, counters=None, sizes=None):
        """counters, sizes: versions() of every layer's connections and network_sizes(), if the caller has them."""
        counters = counters or [versions(a, b) or (None, None) for a, b, _ in layers]
        self.layers = [layer + counter for layer, counter in zip(layers, counters)]
        self.sizes = sizes or network_sizes(n_in, layers)
        self.program = None
        for a, b, gate in layers:
            _index(a, "a", gate.numel())
            _index(b, "b", gate.numel())
        if build:
            self.build()
        else:   # the gates are in this stream's queue; build() may be called on another one
            with N.on_device(layers[0][2]):
                self.gates_ready = torch.cuda.current_stream().record_event()

    gates_ready = None
    counted = None      # number of classes to make a table for along with the program
    layer_by_layer = False      # neither folded nor, all layers or the hidden ones, in one kernel, whatever the classes
    samples = None      # of the pass that it is built for; None: the form for large batches
    limit = None        # samples of a pass from which on that form is wanted and not there

    def folds(self, samples):
        """Whether a pass of so many samples wants the network folded."""
        return max(self.sizes[1:]) > FOLD_ROWS or sum(self.sizes[1:]) * samples >= FOLD_WORK

    def build(self):
        samples, k = self.samples, self.counted      # once: another thread may want another form, and count other classes
        if samples is not None and not self.folds(samples):
            self._keep_whole()
            self.limit = -(-FOLD_WORK // sum(self.sizes[1:]))
            return
        program = self._folded()
        if int(program[3]) * 4 >= 3 * sum(self.sizes[1:]):     # hardly folded: all neurons take less time
            self._keep_whole(program[:4].clone())
            self.limit = None
        else:
            self.order(program, k)

    def _folded(self):
        """Room for the folded program, so far with the number of gates left (word 3)."""
        count = len(self.layers)
        program = torch.empty(N.lib().dl_network_program_words(self.sizes, count), dtype=torch.int32, device=self.layers[0][2].device)
        self._launch(N.lib().dl_network_fold, program)
        return program

    def order(self, program, k=None):
        """The rest of it, and the class table for k."""
        with N.on_device(program):
            N.check_status(N.lib().dl_network_order(self.sizes, len(self.layers), program.data_ptr(), N.stream_of(program)))
        table = None if k is None else self._make_table(program, k)
        # other threads and streams may take program and table from here on: this waits for them
        program._dl_needs = tuple(program[:2].tolist())     # slots, gates of a layer
        program._dl_tables = {} if table is None else {k: table}     # by number of classes, of this program's slots
        program._dl_whole = None
        self.program, self.limit = program, None

    def _keep_whole(self, header=None):
        whole = self._whole()
        program = whole[:4] if header is None else header
        program._dl_whole, program._dl_needs, program._dl_tables, program._dl_stream = whole, None, {}, whole._dl_stream
        self.program = program

    def _whole(self):
        """The program for all neurons, finished."""
        whole = getattr(self.program, '_dl_whole', None)
        if whole is not None:
            return whole
        whole = torch.empty(N.lib().dl_network_whole_words(self.sizes, len(self.layers)), dtype=torch.int32, device=self.layers[0][2].device)
        self._launch(N.lib().dl_network_whole, whole)
        torch.cuda.current_stream(whole.device).synchronize()
        return whole

    def _launch(self, build, program, *scratch):
        """build(connections, gates, sizes, layers, program, scratch, stream)."""
        import ctypes
        count = len(self.layers)
        pointers = [(ctypes.c_void_p * count)(*[layer[i].data_ptr() for layer in self.layers]) for i in range(3)]
        with torch.cuda.device(program.device):
            stream = torch.cuda.current_stream(program.device)
            if self.gates_ready is not None:
                stream.wait_event(self.gates_ready)
            N.check_status(build(*pointers, self.sizes, count, program.data_ptr(), *[t.data_ptr() for t in scratch], stream.cuda_stream))
        program._dl_stream = stream.cuda_stream

    def _table_of(self, program, k, stream):
        layers = len(self.layers)
        table = torch.empty(N.lib().dl_network_table_words(self.sizes, layers, k), dtype=torch.int32, device=program.device)
        N.check_status(N.lib().dl_network_table(program.data_ptr(), self.sizes, layers, k, table.data_ptr(), stream))
        return table

    def _make_table(self, program, k):
        with N.on_device(program):
            stream = N.stream_of(program)
            table = self._table_of(program, k, stream)
        table._dl_stream = stream
        return table

    def table(self, program, k):
        """The class table of a program for k classes; made, and waited for, when k is met first.  Other threads, whose streams wait
        for nothing, see it when it is finished."""
        table = program._dl_tables.get(k)
        if table is None:
            table = self._make_table(program, k)
            torch.cuda.current_stream(table.device).synchronize()
            others = program._dl_tables
            program._dl_tables = {**(others if len(others) < 4 else {}), k: table}
        return table

    def serves(self, x, k):
        """Whether the program is there, has counted k classes before, and takes the rows of x: all that has to be asked of a
        pass that is like an earlier one.  (What the classes' counts need depends on k alone, not on the batch.)"""
        program, limit = self.program, self.limit
        return (program is not None and (limit is None or x.shape[1] * x.element_size() * 8 < limit) and k in getattr(program, '_dl_tables', ()) and x.shape[1] * x.element_size() % 16 == 0
                and x.data_ptr() % 16 == 0 and x.is_contiguous() and x.numel() > 0)

    def matches(self, layers):
        return len(layers) == len(self.layers) and all(
            a is p[0] and b is p[1] and gate is p[2] and p[3] is not None and a._version == p[3] and b._version == p[4]
            for (a, b, gate), p in zip(layers, self.layers))


FOLDED_LAYERS = 32     # layers of a network that can be folded
ONE_KERNEL_ROWS = 1 << 14     # rows of an input or a layer that the one-kernel evaluation takes at most


class FoldedLayers(NetworkProgram):
    """The same for networks of any width (dl_fold_layers): the gates that are left of every layer, and how many they are."""

    def __init__(self, n_in, layers, build=True, counters=None, sizes=None):
        counters = counters or [versions(a, b) or (None, None) for a, b, _ in layers]
        self.layers = [layer + counter for layer, counter in zip(layers, counters)]
        self.sizes = sizes or network_sizes(n_in, layers)
        self.program = None
        self.stream = N.stream_of(layers[0][2])     # the gates are in its queue
        if build:
            self.build()

    def build(self):
        import ctypes
        count = len(self.layers)
        for a, b, gate, _, _ in self.layers:
            _index(a, "a", gate.numel())
            _index(b, "b", gate.numel())
        device = self.layers[0][2].device
        if N.stream_of(self.layers[0][2]) != self.stream:
            torch.cuda.synchronize(device)
        program = torch.empty(N.lib().dl_fold_layers_bytes(self.sizes, count), dtype=torch.uint8, device=device)
        scratch = torch.empty(N.lib().dl_fold_scratch_bytes(self.sizes, count), dtype=torch.uint8, device=device)
        self._launch(N.lib().dl_fold_layers, program, scratch)
        k = self.counted        # once: another thread may count other classes
        table = None if k is None else self._make_table(program, k)
        # other threads and streams may take program and table from here on: this waits for them
        left = scratch[:4 * count].view(torch.int32).tolist()
        program._dl_tables = {} if table is None else {k: table}
        program._dl_left = (ctypes.c_int32 * count)(*left)
        self.rows = sum(left[1:])
        # fewer rows to compute than by whole layers, and at most half as much memory again as two activations of the widest layer
        self.pays = self.rows * 10 <= 9 * sum(self.sizes[1:-1]) and self.rows <= 3 * max(self.sizes[1:])
        self.program = program

    def _table_of(self, program, k, stream):
        layers = len(self.layers)
        table = torch.empty(N.lib().dl_fold_tail_bytes(self.sizes, layers, k), dtype=torch.uint8, device=program.device)
        N.check_status(N.lib().dl_fold_tail(program.data_ptr(), self.sizes, layers, k, table.data_ptr(), stream))
        at = 16 * self.sizes[layers]
        table._dl_longest = int(table[at:at + 4].view(torch.int32))
        return table

    def serves(self, x, k):
        return super().serves(x, k) and self.pays

    def drop(self):
        """What remains of a network that does not pay: that it does not, and whether that is all there is to ask."""
        self.program = ()
        self.layer_by_layer = max(self.sizes[:-1]) > ONE_KERNEL_ROWS


def row_counts(rows):
    import ctypes
    return (ctypes.c_int64 * len(rows))(*rows)


def network_sizes(n_in, layers):
    return row_counts([n_in] + [gate.numel() for _, _, gate in layers])


def eval_network_applicable(x, sizes, batch, k):
    """True when the one-kernel network evaluation takes layers of these sizes on packed words x."""
    if not (x.is_cuda and x.dim() == 2 and x.is_contiguous() and x.dtype in _DTYPE_TO_BITS and x.shape[0] == sizes[0]):
        return False
    return N.lib().dl_eval_network_applicable(x.data_ptr(), sizes, len(sizes) - 1, x.shape[1] * (bits_of(x) // 8), int(batch), int(k)) != 0


def eval_network(x, network, batch, k=None):
    """All layers of a NetworkProgram on packed words x in one kernel: int32 [batch, k] class counts, or without k the last
    layer's rows as packed words."""
    _need(x.is_cuda and x.dim() == 2 and x.is_contiguous(), "x must be a contiguous 2-D CUDA tensor")
    sizes, program, words = network.sizes, network.program, x.shape[1]     # another thread may build the same program once more
    _need(x.shape[0] == sizes[0] and x.device == program.device, "x does not fit the network")
    row_bytes = words * (bits_of(x) // 8)
    if k is None:
        out = torch.empty((sizes[len(sizes) - 1], words), dtype=x.dtype, device=x.device)
    else:
        out = torch.empty((int(batch), int(k)), dtype=torch.int32, device=x.device)
    with N.on_device(x):
        if program._dl_whole is None and program._dl_needs is None:
            network.order(network._folded())
            program = network.program
        whole = program._dl_whole
        if whole is not None and k is not None:
            program._dl_tables.setdefault(int(k))       # counts these without a table
        table = None if k is None or whole is not None else network.table(program, int(k))
        stream = N.stream_of(x)
        for t in (program, table, whole):
            if t is not None and stream != t._dl_stream:
                t.record_stream(torch.cuda.current_stream(x.device))
        if whole is not None:
            N.check(N.lib().dl_eval_whole(x.data_ptr(), whole.data_ptr(), sizes, len(sizes) - 1, 0 if k is None else out.data_ptr(),
                                          out.data_ptr() if k is None else 0, row_bytes, int(batch), 1 if k is None else int(k), stream))
            return out
        N.check(N.lib().dl_eval_network_sized(x.data_ptr(), program.data_ptr(), sizes, len(sizes) - 1, *program._dl_needs,
                                              N.ptr(table), 0 if k is None else out.data_ptr(), out.data_ptr() if k is None else 0, row_bytes,
                                              int(batch), 1 if k is None else int(k), stream))
    return out


def eval_folded_applicable(x, sizes):
    """True when a network of these sizes on packed words x can be folded: more than one layer, and the sizes of dl_fold_layers."""
    return (x.is_cuda and x.dim() == 2 and x.is_contiguous() and x.dtype in _DTYPE_TO_BITS and x.shape[0] == sizes[0] and x.shape[1] > 0
            and 2 < len(sizes) <= FOLDED_LAYERS + 1 and 0 < min(sizes) and sum(sizes) < 1 << 27)


def eval_folded_counts_applicable(x, sizes, rows, k):
    """True when eval_folded counts classes of these rows of a network with `rows` gates left: whole units of 16 bytes, whose places
    in a buffer fit 32 bits."""
    row_bytes = x.shape[1] * x.element_size()
    return k > 0 and sizes[len(sizes) - 1] % k == 0 and row_bytes % 16 == 0 and x.data_ptr() % 16 == 0 and max(rows, sizes[0]) * row_bytes < 1 << 35


def eval_folded(x, network, batch, k=None):
    """All layers of a FoldedLayers on packed words x: int32 [batch, k] class counts, or without k the last layer's rows as
    packed words."""
    _need(x.is_cuda and x.dim() == 2 and x.is_contiguous(), "x must be a contiguous 2-D CUDA tensor")
    sizes, program, words = network.sizes, network.program, x.shape[1]
    _need(x.shape[0] == sizes[0] and x.device == program.device, "x does not fit the network")
    row_bytes = words * (bits_of(x) // 8)
    pool = torch.empty((sum(program._dl_left[1:]), words), dtype=x.dtype, device=x.device)
    if k is None:
        out = torch.empty((sizes[len(sizes) - 1], words), dtype=x.dtype, device=x.device)
    else:
        out = torch.empty((int(batch), int(k)), dtype=torch.int32, device=x.device)
    with N.on_device(x):
        table = None if k is None else network.table(program, int(k))
        stream = N.stream_of(x)
        for t in (program, table):
            if t is not None and stream != t._dl_stream:
                t.record_stream(torch.cuda.current_stream(x.device))
        N.check(N.lib().dl_eval_folded(x.data_ptr(), program.data_ptr(), sizes, program._dl_left, len(sizes) - 1, pool.data_ptr(),
                                       N.ptr(table), 0 if k is None else table._dl_longest, 0 if k is None else out.data_ptr(), out.data_ptr() if k is None else 0, row_bytes, int(batch),
                                       1 if k is None else int(k), stream))
    return out


# ------------------------------------------------------------------------------------------------
# float GroupSum
# ------------------------------------------------------------------------------------------------

_workspaces = {}


def _groupsum_workspace(device, stream, nbytes):
    """Zero-initialised scratch for dl_groupsum_f32, grown on demand.  The kernel leaves the counters at
    zero, so a buffer is cleared only when it is created.  Eager calls use one buffer per (device, stream).
    Calls made while a CUDA graph is being captured share one buffer per device that is created by the first
    eager call on that device (warm-up steps), so that a captured step contains no allocation and no memset;
    graphs replayed concurrently on different streams must therefore not both contain a GroupSum."""
    want = max(nbytes, 1 << 20)
    graph_key = (device, "graph")
    capturing = torch.cuda.is_current_stream_capturing()
    if not capturing:
        gws = _workspaces.get(graph_key)
        if gws is None or gws.numel() < want:
            _workspaces[graph_key] = torch.zeros(want, dtype=torch.uint8, device=device)
    key = graph_key if capturing else (device, stream)
    ws = _workspaces.get(key)
    if ws is None or ws.numel() < nbytes:
        ws = torch.zeros(want, dtype=torch.uint8, device=device)
        _workspaces[key] = ws
    return ws


def groupsum_workspace(x, k):
    """Scratch for the sums of x [batch, n] in k classes, by a call on the current stream."""
    return _groupsum_workspace(x.device, N.stream_of(x), N.lib().dl_groupsum_workspace_bytes(x.shape[1], x.shape[0], k))


def groupsum(x, k, tau):
    """feature-major x [n, batch] -> [batch, k] = per-class row sums / tau."""
    _f32_matrix(x, "x")
    n, batch = x.shape
    k = int(k)
    _need(k > 0 and n % k == 0, "n (%d) must be divisible by k (%d)" % (n, k))
    out = x.new_empty((batch, k))
    with N.on_device(x):
        stream = N.stream_of(x)
        ws = _groupsum_workspace(x.device, stream, N.lib().dl_groupsum_workspace_bytes(n, batch, k))
        N.check(N.lib().dl_groupsum_f32(x.data_ptr(), out.data_ptr(), ws.data_ptr(), n, batch, k, float(tau), stream))
    return out


_HEAD_COUNTERS = {}


def groupsum_cross_entropy_applicable(n, batch, k):
    return N.lib().dl_groupsum_cross_entropy_applicable(int(n), int(batch), int(k)) == 1


def groupsum_cross_entropy(x, target, k, tau):
    """Head of a training step in one kernel.  feature-major x [n, batch], int64 target [batch] ->
    (loss scalar, scores [batch, k], grad_classes [k, batch]); grad_classes is the gradient of the mean cross-entropy
    loss w.r.t. every output row of a class, for logic_backward_w / logic_backward_x with rows_per_class = n / k."""
    _f32_matrix(x, "x")
    n, batch = x.shape
    k = int(k)
    _need(k > 0 and n % k == 0, "n (%d) must be divisible by k (%d)" % (n, k))
    _need(target.is_cuda and target.dtype == torch.int64 and target.dim() == 1 and target.is_contiguous()
          and target.shape[0] == batch and target.device == x.device, "target must be a contiguous int64 [batch] CUDA tensor")
    _need(groupsum_cross_entropy_applicable(n, batch, k), "classes of %d rows are outside the fused kernel's range" % (n // k))
    scores = x.new_empty((batch, k))
    loss = torch.empty((), dtype=torch.float32, device=x.device)
    grad_classes = x.new_empty((k, batch))
    counter = _HEAD_COUNTERS.get(x.device)
    if counter is None:
        counter = _HEAD_COUNTERS[x.device] = torch.zeros(1, dtype=torch.int32, device=x.device)
    with N.on_device(x):
        N.check(N.lib().dl_groupsum_cross_entropy_f32(x.data_ptr(), target.data_ptr(), scores.data_ptr(), loss.data_ptr(),
                                                      grad_classes.data_ptr(), counter.data_ptr(), n, batch, k, float(tau),
                                                      N.stream_of(x)))
    return loss, scores, grad_classes


def forward_head_applicable(n_out, batch, k):
    """True when logic_forward_head takes these sizes: classes at least as long as a forward CTA's run of rows."""
    return N.lib().dl_forward_class_sums_rows(int(n_out), int(batch), int(k)) > 0


def logic_forward_head(x, a, b, w, target, k, tau, w_mode=W_LOGITS):
    """Last layer + GroupSum(k, tau) + mean cross-entropy in two kernels that never store the layer's output:
    (loss scalar, scores [batch, k], grad_classes [k, batch], coef [n_out, 4]).  The forward kernel's CTAs add up
    their rows per class; a small second kernel adds those pieces in a fixed order and does the loss.  grad_classes
    is for logic_backward_w / logic_backward_x with rows_per_class = n_out / k."""
    _f32_matrix(x, "x")
    _f32_matrix(w, "w")
    n_in, batch = x.shape
    n_out, k = w.shape[0], int(k)
    _need(w.shape[1] == 16, "w must be [n_out, 16]")
    _index(a, "a", n_out)
    _index(b, "b", n_out)
    _need(k > 0 and n_out % k == 0, "n_out (%d) must be divisible by k (%d)" % (n_out, k))
    _need(target.is_cuda and target.dtype == torch.int64 and target.dim() == 1 and target.is_contiguous()
          and target.shape[0] == batch and target.device == x.device, "target must be a contiguous int64 [batch] CUDA tensor")
    lib = N.lib()
    rows = lib.dl_forward_class_sums_rows(n_out, batch, k)
    _need(rows > 0, "classes of %d rows are shorter than a forward CTA's run of rows" % (n_out // k))
    sums = x.new_empty((rows, batch))
    coef = x.new_empty((n_out, 4))
    scores = x.new_empty((batch, k))
    loss = torch.empty((), dtype=torch.float32, device=x.device)
    grad_classes = x.new_empty((k, batch))
    counter = _HEAD_COUNTERS.get(x.device)
    if counter is None:
        counter = _HEAD_COUNTERS[x.device] = torch.zeros(1, dtype=torch.int32, device=x.device)
    with N.on_device(x):
        st = N.stream_of(x)
        N.check(lib.dl_forward_class_sums_f32(x.data_ptr(), a.data_ptr(), b.data_ptr(), w.data_ptr(), w_mode, sums.data_ptr(),
                                              coef.data_ptr(), n_in, n_out, batch, k, N.LAUNCH_OVERLAP_SETUP, st))
        N.check(lib.dl_class_sums_cross_entropy_f32(sums.data_ptr(), target.data_ptr(), scores.data_ptr(), loss.data_ptr(),
                                                    grad_classes.data_ptr(), counter.data_ptr(), n_out, batch, k,
                                                    lib.dl_forward_class_sums_run(batch), float(tau), st))
    return loss, scores, grad_classes, coef


def groupsum_backward(grad_out, n, tau):
    """[batch, k] -> feature-major [n, batch] with grad_x[i,:] = grad_out[:, i // (n/k)] / tau."""
    _f32_matrix(grad_out, "grad_out")
    batch, k = grad_out.shape
    gx = torch.empty((n, batch), dtype=torch.float32, device=grad_out.device)
    with N.on_device(grad_out):
        N.check(N.lib().dl_groupsum_backward_f32(grad_out.data_ptr(), gx.data_ptr(), n, batch, k, float(tau),
                                                 N.stream_of(grad_out)))
    return gx
