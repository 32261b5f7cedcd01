"""The loss head over long classes, whose sums eight CTAs share: scores, loss and gradient against 64-bit torch."""
import pytest
import torch

from difflogic_b200 import functional, ops
from tests.helpers import assert_forward_close, assert_grad_close

pytestmark = pytest.mark.gpu


# (n_out, k, batch): 64 and 63 runs of 32 rows per class, classes that end inside a run, several blocks of columns, so many
# (columns, class) pairs that one CTA each will do
@pytest.mark.parametrize("n_out,k,batch", [(2 * 2048, 2, 200), (2 * 1984, 2, 200), (3 * 3001, 3, 333), (20000, 1, 130), (30000, 10, 1900), (2 * 10000, 2, 256)])
def test_head(n_out, k, batch):
    g = torch.Generator().manual_seed(n_out)
    n_in, tau = 50, 20.0
    x, w = torch.rand(n_in, batch, generator=g), torch.randn(n_out, 16, generator=g)
    a, b = torch.randint(0, n_in, (2, n_out), generator=g)
    target = torch.randint(0, k, (batch,), generator=g)
    mix = torch.softmax(w.double(), 1)
    y = functional.bin_op_s(x.double()[a].t(), x.double()[b].t(), mix)
    ref = (y.reshape(batch, k, -1).sum(-1) / tau).requires_grad_()
    loss_ref = torch.nn.functional.cross_entropy(ref, target)
    loss_ref.backward()
    for _ in range(2):      # the ticket is back at zero
        loss, scores, grad_classes, _ = ops.logic_forward_head(x.cuda(), a.cuda(), b.cuda(), w.cuda(), target.cuda(), k, tau)
        assert_forward_close(scores, ref, "scores")
        assert abs(loss.item() - loss_ref.item()) <= 1e-5 * max(1.0, ref.abs().max().item())
        if k > 1:
            assert_grad_close(grad_classes.t() * tau, ref.grad, "grad")
    if batch % 128 == 0:    # the order of the additions does not depend on how many CTAs share them: 19 blocks of columns more
        wide = torch.cat([x] + [torch.rand(n_in, 128 * 19, generator=g)] * 4, 1)
        fill = torch.zeros(wide.shape[1] - batch, dtype=torch.int64)
        _, more, _, _ = ops.logic_forward_head(wide.cuda(), a.cuda(), b.cuda(), w.cuda(), torch.cat([target, fill]).cuda(), k, tau)
        assert torch.equal(more[:batch], scores)
