"""Layers and batches that leave the GPU short of CTAs take fewer rows per CTA and more lanes per neuron: forward and weight gradient
against 64-bit torch around the sizes where the kernels change shape."""
import pytest
import torch

from difflogic_b200 import functional, ops
from tests.helpers import assert_forward_close, assert_grad_close

pytestmark = pytest.mark.gpu


# 148 CTAs: 9472 neurons of 4 lanes, 2368 of 16; 4 passes of 64 row groups
@pytest.mark.parametrize("batch", [1, 3, 4, 16, 17, 32, 33, 64, 260])
@pytest.mark.parametrize("n_out", [1, 15, 65, 1000, 2367, 2369, 9473])
def test_forward_and_weight_gradient(n_out, batch):
    g = torch.Generator().manual_seed(n_out * 1000 + batch)
    n_in = min(300, 2 * n_out)
    x, w, gy = torch.rand(n_in, batch, generator=g), torch.randn(n_out, 16, generator=g), torch.randn(n_out, batch, generator=g)
    a, b = torch.randint(0, n_in, (2, n_out), generator=g)
    xd, wd = x.double(), w.double().requires_grad_()
    mix = torch.softmax(wd, 1)
    ref = functional.bin_op_s(xd[a].t(), xd[b].t(), mix).t()
    ref.backward(gy.double())
    y, _ = ops.logic_forward(x.cuda(), a.cuda(), b.cuda(), w.cuda())
    gw = ops.logic_backward_w(x.cuda(), a.cuda(), b.cuda(), gy.cuda(), w.cuda(), ops.W_LOGITS)
    assert_forward_close(y, ref, "y")
    assert_grad_close(gw, wd.grad, "grad_w")
