"""The staged backward kernel of the walk (rows copied into shared memory ahead of their step) against a float64 restatement, forced at
sizes where it can go wrong: parts of one turn of eight steps, several turns, more parts than the walk fills, a walk that ends inside a
turn, one column block that is not full and up to sixteen of them, more column blocks than turns wait for one epilogue (8), few classes."""
import pytest
import torch

from difflogic_b200 import _native as N
from difflogic_b200 import ops
from tests.helpers import assert_grad_close
from tests.test_gpu_walk import _connections, _reference

pytestmark = pytest.mark.gpu


def assert_adam(w, grad, start, step, w_got, moments, lr=0.01, beta1=0.9, beta2=0.999, eps=1e-8):
    """Weights and both moments of every neuron against the step in 64 bits from the same gradient and float constants.  Moments: one
    rounding of each product and sum (2^-24 each).  Weights: one of the sum, and of the update 1 - beta2^step, in which the last place of a
    power close to 1 is 6e-8 / 5e-3 = 1.2e-5 at step 5; twice that for a power that is two places off."""
    beta1, beta2, lr, eps = (float(torch.tensor(v)) for v in (beta1, beta2, lr, eps))
    w, grad, (m, v) = w.double().flatten(), grad.double().flatten(), [t.double() for t in start]
    m_ref, v_ref = m + (grad - m) * (1 - beta1), v * beta2 + grad * grad * (1 - beta2)
    update = lr / (1 - beta1 ** step) * m_ref / (v_ref.sqrt() / (1 - beta2 ** step) ** 0.5 + eps)
    m_got, v_got = (t.cpu().double() for t in moments)
    assert bool(((m_got - m_ref).abs() <= 2 ** -22 * (m.abs() + grad.abs())).all())
    assert bool(((v_got - v_ref).abs() <= 2 ** -22 * v_ref).all())
    assert bool(((w_got.cpu().double().flatten() - (w - update)).abs() <= 3e-5 * update.abs() + 2 ** -22 * m.abs() * lr / v_ref.sqrt() + 2 ** -23 * w.abs()).all())


@pytest.mark.parametrize("batch", [4, 36, 128, 132, 256, 640, 1024, 1028, 1160, 2048])
@pytest.mark.parametrize("case,classes", [(("square", 1, 1), 1), (("square", 9, 9), 9), (("square", 2500, 2500), 5), (("square", 19000, 19000), 19000),
                                          (("paths", 150, 70), 70), (("loops", 70, 65), 13), (("any", 40, 5000), 5000)])
def test_staged_backward(case, classes, batch):
    kind, n_in, n_out = case
    if n_out * batch > 10_000_000:
        batch = batch // 16 * 4 or 4                        # the oracle's memory and time
    a, b = _connections(*case)
    g = torch.Generator().manual_seed(batch)
    x, w, gyc = torch.rand(n_in, batch, generator=g), torch.randn(n_out, 16, generator=g), torch.randn(classes, batch, generator=g)
    _, gx_ref, gw_ref = _reference(x, a, b, w, gyc.repeat_interleave(n_out // classes, 0), 1.5)
    walk = ops.build_walk(a.cuda(), b.cuda(), n_in)
    xd, wd, gyd, coef = x.cuda(), w.cuda(), gyc.cuda(), ops.logic_coefs(w.cuda())
    for want_x in {False, walk.complete}:
        start = [0.1 * torch.randn(n_out * 16, generator=g), 0.01 * torch.rand(n_out * 16, generator=g)]
        moments = [t.cuda() for t in start]
        state, w2 = torch.tensor([4, 0], dtype=torch.int32, device="cuda"), wd.clone()      # the fifth step
        with N.tuning(N.TUNE_WALK_KERNEL, 2):
            gx, gw = ops.logic_backward_walk(xd, gyd, coef, wd, walk, 1.5, want_grad_x=want_x, rows_per_class=n_out // classes)
            gx2, _ = ops.logic_backward_walk(xd, gyd, coef, w2, walk, 1.5, want_grad_x=want_x, rows_per_class=n_out // classes,
                                             adam=dict(exp_avg=moments[0], exp_avg_sq=moments[1], state=state, lr=0.01, beta1=0.9, beta2=0.999,
                                                       eps=1e-8, grad_scale=0.5))
        with N.tuning(N.TUNE_WALK_KERNEL, 1):
            gx_register, _ = ops.logic_backward_walk(xd, gyd, coef, wd, walk, 1.5, want_grad_x=want_x, rows_per_class=n_out // classes)
        assert_grad_close(gw, gw_ref, "grad_w")
        assert state.tolist() == [5, 0]
        assert_adam(w, gw.cpu() * 0.5, start, 5, w2, moments)
        if want_x:
            assert_grad_close(gx, gx_ref, "grad_x")
            assert torch.equal(gx, gx_register) and torch.equal(gx2, gx)      # the same two terms, wherever the walk is cut


def test_its_sums_are_as_accurate():
    """Against 64 bits no further off than the register kernel's (both are a few roundings; 1.5 as for the gather kernel's)."""
    n, batch = 4000, 1024
    a, b = _connections("square", n, n)
    g = torch.Generator().manual_seed(batch)
    x, w, gy = torch.rand(n, batch, generator=g), torch.randn(n, 16, generator=g), torch.randn(n, batch, generator=g)
    want = _reference(x, a, b, w, gy, 1.0)[2]
    walk, coef = ops.build_walk(a.cuda(), b.cuda(), n), ops.logic_coefs(w.cuda())
    error = []
    for kernel in (1, 2):
        with N.tuning(N.TUNE_WALK_KERNEL, kernel):
            got = ops.logic_backward_walk(x.cuda(), gy.cuda(), coef, w.cuda(), walk)[1]
        error.append(float((got.cpu().double() - want).norm() / want.norm()))
    assert error[1] <= 1.5 * error[0], error
