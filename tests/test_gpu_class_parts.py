"""Last layer and class counts in one kernel for classes longer than a cluster's counters (2040 gates): counted in parts."""
import pytest
import torch

from difflogic_b200 import _native as N
from difflogic_b200 import ops

pytestmark = pytest.mark.gpu


# (n_in, k, gates per class, words, bits, pad_len): just over the limit, a prime, one class, many parts; one block of columns,
# several, a ragged last one
@pytest.mark.parametrize("n_in,k,m,words,bits,pad_len", [(64, 3, 2041, 64, 64, 0), (200, 2, 4099, 132, 32, 5), (3000, 1, 30001, 64, 64, 63),
                                                         (90, 10, 2500, 532, 64, 0), (500, 7, 8160, 272, 16, 1), (64, 2, 32000, 2048, 8, 0)])
def test_counts_in_parts(n_in, k, m, words, bits, pad_len):
    g = torch.Generator(device="cuda").manual_seed(m)
    n_out = k * m
    x = torch.randint(-2 ** 63, 2 ** 63 - 1, (n_in, words * bits // 64), device="cuda", generator=g).view(getattr(torch, "int%d" % bits))
    a, b = torch.randint(0, n_in, (2, n_out), device="cuda", generator=g)
    gate = torch.randint(0, 16, (n_out,), device="cuda", generator=g).to(torch.uint8)
    assert ops.eval_groupbitsum_parts_applicable(x, n_out, k) and not ops.eval_groupbitsum_applicable(x, n_out, k)
    want = ops.groupbitsum(ops.eval_packed(x, a, b, gate), pad_len, k)
    for _ in range(2):
        assert torch.equal(ops.eval_groupbitsum(x, a, b, gate, pad_len, k, parts=True), want)
    assert N.lib().dl_async_error() == 0


def test_range():
    x = torch.zeros(64, 64, dtype=torch.int64, device="cuda")
    assert ops.eval_groupbitsum_parts_applicable(x, 4082, 2)
    assert not ops.eval_groupbitsum_parts_applicable(x, 4080, 2)                        # the plain kernel takes it
    assert not ops.eval_groupbitsum_parts_applicable(x, 4083, 2)                        # not divisible
    assert not ops.eval_groupbitsum_parts_applicable(x[:, :32].contiguous(), 4082, 2)   # rows of 256 bytes
