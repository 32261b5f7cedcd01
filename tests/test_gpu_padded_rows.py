"""Batches that do not fill whole 16-byte units: rows are padded inside PackBitsTensor, which must show neither in `.t` nor in
the counts.  Row lengths on both sides of the staged kernels' 512-byte limit, every word width, fused and unfused tails."""
import pytest
import torch

import difflogic_b200 as D
from difflogic_b200.compiled_model import CompiledLogicNet

pytestmark = pytest.mark.gpu


def _hidden(model, xb):
    h = xb
    for layer in [l for l in model if isinstance(l, D.LogicLayer)]:
        gate, (a, b) = layer.weights.detach().argmax(1), layer.indices
        t00, t01, t10, t11 = [((gate >> s) & 1).bool() for s in (3, 2, 1, 0)]
        A, B = h[:, a], h[:, b]
        h = torch.where(A, torch.where(B, t11, t10), torch.where(B, t01, t00))
    return h


@pytest.mark.parametrize("bits", [8, 16, 32, 64])
@pytest.mark.parametrize("batch", [1, 7, 65, 127, 128, 129, 4000, 4096, 4100, 10007])
@pytest.mark.parametrize("n_in,width,k", [(40, 60, 2), (33, 640, 10), (24, 4200, 2)])   # classes of 30, 64 and 2100 rows
def test_ragged_batches(n_in, width, k, batch, bits):
    torch.manual_seed(batch + width)
    model = torch.nn.Sequential(torch.nn.Flatten(), D.LogicLayer(n_in, width), D.LogicLayer(width, width), D.GroupSum(k)).eval()
    with torch.no_grad():
        xb = torch.rand(batch, n_in, device="cuda") < 0.4
        hidden = _hidden(model, xb)
        want = hidden.reshape(batch, k, -1).sum(-1).int()
        p = D.PackBitsTensor(xb, bit_count=bits)
        assert torch.equal(model(p), want)
        words = -(-batch // bits)
        assert p.t.shape == (width, words) and p.t.is_contiguous() and p.pad_len == words * bits - batch
        lanes = torch.arange(bits, device="cuda")
        unpacked = ((p.t.to(torch.int64).unsqueeze(-1) >> lanes) & 1).reshape(width, -1)[:, :batch].T.bool()
        assert torch.equal(unpacked, hidden)
        assert torch.equal(p.group_sum(k), want)       # from the plain words that `.t` has left
        assert torch.equal(model(D.PackBitsTensor.from_packed(D.PackBitsTensor(xb, bit_count=bits).t, p.pad_len)), want)
        px = torch.randint(0, 256, (batch, n_in // 3 + 8), dtype=torch.uint8, device="cuda")
        q = D.PackBitsTensor.from_uint8_thresholds(px, (63, 127, 191), bit_count=bits)
        thermo = torch.cat([px > t for t in (63, 127, 191)], 1)
        assert torch.equal(q.t, D.PackBitsTensor(thermo, bit_count=bits).t)
        net = CompiledLogicNet(model, device="cuda", num_bits=bits)
        net.compile()
        assert torch.equal(net(xb), want)
