"""Both tiles of the packers (a thread takes 8 or 32 samples) against torch: features and batches around the tiles' edges, rows
and sources at every alignment."""
import pytest
import torch

from difflogic_b200 import ops

pytestmark = pytest.mark.gpu

# (features, batch): the first group is small enough for the tile of 256 features x 64 samples, the second large enough for the one of
# 64 x 1024: 592 such tiles for up to 128 features, 2368 for more (several blocks of features, whole and ragged, aligned and not)
SIZES = [(1, 1), (7, 63), (8, 64), (9, 65), (63, 7), (64, 128), (65, 129), (255, 2047), (256, 2048), (257, 2049), (784, 100), (785, 1000),
         (9, 1300001), (64, 1212416), (70, 620003), (1000, 152000), (1003, 152001), (2048, 76000)]


def _pack(bits, word_bits):
    batch, n = bits.shape
    words = -(-batch // word_bits)
    rows = torch.zeros((n, words * word_bits), dtype=torch.uint8, device=bits.device)
    rows[:, :batch] = bits.t()
    weights = (1 << torch.arange(8, device=bits.device)).to(torch.uint8)
    return (rows.view(n, -1, 8) * weights).sum(-1, dtype=torch.uint8)


def _bytes(words, row_bytes):
    return words.view(torch.uint8).reshape(words.shape[0], -1)[:, :row_bytes]


@pytest.mark.parametrize("offset", [0, 1, 4, 8])
@pytest.mark.parametrize("n,batch", SIZES)
def test_pack(n, batch, offset):
    g = torch.Generator(device="cuda").manual_seed(n + batch)
    flat = torch.randint(0, 256, (n * batch + offset,), dtype=torch.uint8, device="cuda", generator=g)
    x = flat[offset:].view(batch, n)                     # the source's first byte at every alignment
    above = x > 100
    flags = torch.empty_like(flat).copy_((flat > 100))[offset:].view(batch, n).view(torch.bool)
    for padded, bits in ((True, 32), (False, 8), (False, 64)):
        got, pad = ops.packbits_batch_major(flags, bits, padded=padded)
        want = _pack(above, 128 if padded else bits)
        assert torch.equal(_bytes(got, want.shape[1]), want) and pad == -batch % bits
    for thresholds in ((100,), (3, 100), (0, 100, 255), (1, 2, 3, 100, 200)) if batch * n < 10_000_000 else ((10, 100, 200),):
        got, _ = ops.threshold_packbits_batch_major(x, thresholds, 16)
        for i, t in enumerate(thresholds):
            want = _pack(x > t, 16)
            assert torch.equal(_bytes(got[i * n:(i + 1) * n], want.shape[1]), want)
