"""The kernels that walk the connection graph against a float64 restatement of the layer, at the sizes where they can go wrong:
rows shorter and longer than a lane group's reach, one and several column blocks, chunks that end inside a walk, open and
closed walks, neurons wired twice to one input, inputs that nobody reads."""
import pytest
import torch

from difflogic_b200 import ops
from tests.helpers import assert_forward_close, assert_grad_close

pytestmark = pytest.mark.gpu


def _square(n, seed):
    g = torch.Generator().manual_seed(seed)
    slots = torch.randperm(2 * n, generator=g) % n
    slots = torch.randperm(n, generator=g)[slots].reshape(2, n)
    return slots[0].contiguous(), slots[1].contiguous()


def _connections(kind, n_in, n_out):
    g = torch.Generator().manual_seed(n_in * 7 + n_out)
    if kind == "square":
        return _square(n_in, n_out)
    if kind == "loops":                      # every neuron reads one input twice; the inputs beyond n_out feed nobody
        a = torch.arange(n_out)
        return a, a.clone()
    if kind == "paths":                      # every input feeds at most one neuron
        p = torch.randperm(n_in, generator=g)[:2 * n_out].reshape(2, n_out)
        return p[0].contiguous(), p[1].contiguous()
    return torch.randint(0, n_in, (n_out,), generator=g), torch.randint(0, n_in, (n_out,), generator=g)


def _reference(x, a, b, w, gy, scale):
    x, w = x.double().requires_grad_(), w.double().requires_grad_()
    p = torch.softmax(w, -1)
    ids = torch.arange(16)
    t00, t01, t10, t11 = [((ids >> s) & 1).double() for s in (3, 2, 1, 0)]
    c0, ca, cb, cab = p @ t00, p @ (t10 - t00), p @ (t01 - t00), p @ (t00 - t01 - t10 + t11)
    A, B = x[a], x[b]
    y = c0[:, None] + ca[:, None] * A + cb[:, None] * B + cab[:, None] * A * B
    y.backward(gy.double())
    return y.detach(), x.grad * scale, w.grad


CASES = [("square", 1, 1), ("square", 2, 2), ("square", 63, 63), ("square", 64, 64), ("square", 200, 200), ("square", 1030, 1030),
         ("loops", 70, 65), ("paths", 150, 70), ("any", 9, 300), ("any", 300, 310)]


@pytest.mark.parametrize("batch", [1, 3, 32, 33, 61, 64, 65, 75, 100, 128, 129, 256, 260, 500, 1024, 1027, 2180])
@pytest.mark.parametrize("case", CASES)
def test_walk_kernels_match_the_layer(case, batch):
    kind, n_in, n_out = case
    a, b = _connections(*case)
    g = torch.Generator().manual_seed(batch)
    x = torch.rand(n_in, batch, generator=g)
    w = torch.randn(n_out, 16, generator=g)
    classes = 5 if n_out % 5 == 0 and kind == "square" else n_out    # one gradient row per class, or one per neuron
    gyc = torch.randn(classes, batch, generator=g)
    gy = gyc.repeat_interleave(n_out // classes, 0)
    walk = ops.build_walk(a.cuda(), b.cuda(), n_in)
    degree = torch.bincount(torch.cat([a, b]), minlength=n_in)
    assert walk[1] == bool((degree <= 2).all())
    y_ref, gx_ref, gw_ref = _reference(x, a, b, w, gy, 1.5)
    xd, wd = x.cuda(), w.cuda()
    y, coef = ops.logic_forward_walk(xd, wd, walk, want_coef=True)
    assert_forward_close(y, y_ref, "forward")
    y_arg, _ = ops.logic_forward_walk(xd, wd, walk, ops.W_ARGMAX)
    assert torch.equal(y_arg, ops.logic_forward(xd, a.cuda(), b.cuda(), wd, ops.W_ARGMAX)[0])
    gx, gw = ops.logic_backward_walk(xd, gyc.cuda(), coef, wd, walk, 1.5, want_grad_x=walk[1], rows_per_class=n_out // classes)
    assert_grad_close(gw, gw_ref, "grad_w")
    if walk[1]:
        assert_grad_close(gx, gx_ref, "grad_x")
    # Adam in the epilogue: the same update as the gather kernel's epilogue, given gradients that differ by rounding only.
    # A first step moves every weight by lr * g / (|g| + eps): where |g| is large beside its error (1e-4 of the largest) the
    # two moves agree to lr * 1e-4 * max|g| / |g|.
    for want_x in {False, walk[1]}:                 # with grad_x: what a hidden layer's training step runs
        state = torch.zeros(2, dtype=torch.int32, device="cuda")
        w2, m, v = wd.clone(), torch.zeros(n_out * 16, device="cuda"), torch.zeros(n_out * 16, device="cuda")
        gx, _ = ops.logic_backward_walk(xd, gyc.cuda(), coef, w2, walk, 1.5, want_grad_x=want_x, rows_per_class=n_out // classes,
                                        adam=dict(exp_avg=m, exp_avg_sq=v, state=state, lr=0.01, beta1=0.9, beta2=0.999, eps=1e-8,
                                                  grad_scale=1.0))
        assert state.tolist() == [1, 0]
        if want_x:
            assert_grad_close(gx, gx_ref, "grad_x beside Adam")
        assert_grad_close(m.view(n_out, 16) * 10, gw_ref, "first moment")
        big = gw_ref.abs() > 1e-2 * gw_ref.abs().max()
        moved = (wd - w2).cpu().double() / 0.01
        assert bool(((moved - gw_ref.sign()).abs()[big] <= 2e-2).all())


def test_a_bad_connection_gives_no_walk():
    a = torch.tensor([0, 1, 5]).cuda()
    assert ops.build_walk(a, a, 5) is None


@pytest.mark.parametrize("batch", [1, 31, 64, 75, 128, 131, 1024, 1027])
@pytest.mark.parametrize("case", CASES)
def test_both_routes_give_the_same_bits(case, batch):
    """A layer may take the walk or the gather kernels from one call to the next: outputs and coefficients are the same to the bit,
    also where rows hold infinities and NaN.  (The gradients' terms are added in another order.)"""
    kind, n_in, n_out = case
    a, b = (t.cuda() for t in _connections(*case))
    g = torch.Generator().manual_seed(batch + 1)
    x = torch.rand(n_in, batch, generator=g).cuda()
    w = torch.randn(n_out, 16, generator=g).cuda()
    walk = ops.build_walk(a, b, n_in)
    for special in (None, float("inf"), float("nan")):
        if special is not None:
            x[::5, ::3] = special
        for mode in (ops.W_LOGITS, ops.W_ARGMAX):
            y, coef = ops.logic_forward_walk(x, w, walk, mode, want_coef=True)
            y_gather, coef_gather = ops.logic_forward(x, a, b, w, mode, want_coef=True)
            assert torch.equal(coef, coef_gather) and torch.allclose(y, y_gather, rtol=0, atol=0, equal_nan=True)


@pytest.mark.parametrize("batch", [75, 128, 1024])
def test_weight_gradients_are_as_accurate_along_the_walk(batch):
    """Their error against 64 bits is not larger than that of the gather kernel's sums (both are a few roundings; 1.5 allows for
    the difference between two samples of them)."""
    n = 4000
    a, b = _square(n, 11)
    g = torch.Generator().manual_seed(batch)
    x, w, gy = torch.rand(n, batch, generator=g), torch.randn(n, 16, generator=g), torch.randn(n, batch, generator=g)
    want = _reference(x, a, b, w, gy, 1.0)[2]
    xd, wd, gyd, ad, bd = x.cuda(), w.cuda(), gy.cuda(), a.cuda(), b.cuda()
    walk = ops.build_walk(ad, bd, n)
    coef = ops.logic_coefs(wd, ops.W_LOGITS)

    def error(got):
        return float((got.cpu().double() - want).norm() / want.norm())
    along = error(ops.logic_backward_walk(xd, gyd, coef, wd, walk)[1])
    gathered = error(ops.logic_backward_w(xd, ad, bd, gyd, wd, ops.W_LOGITS))
    assert along <= 1.5 * gathered, (along, gathered)


def test_edited_connections_are_followed_at_every_batch_size():
    """In-place writes and assignments of `indices`: the walk (large batches) and the gather kernels (small ones) use the same."""
    import difflogic_b200 as D
    torch.manual_seed(2)
    n = 12000
    layer = D.LogicLayer(n, n).eval()
    x = (torch.rand(200, n, device="cuda") < 0.5).float()

    def check():
        want = ops.logic_forward(x.t().contiguous(), *layer.indices, layer.weights.detach(), ops.W_ARGMAX)[0].t()
        with torch.no_grad():
            for _ in range(3):
                assert torch.equal(layer(x), want) and torch.equal(layer(x[:10]), want[:10])
    check()
    layer.indices[0].copy_(layer.indices[0].flip(0))
    check()
    layer.indices = (layer.indices[0], layer.indices[1].flip(0).contiguous())
    check()
    layer.set_connections(layer.indices[1].clone(), layer.indices[0].clone())
    check()
