"""Pad lengths beyond the last word are refused, whatever the rows' length; only rows that the package itself has padded to 16 bytes
leave out whole words."""
import pytest
import torch

from difflogic_b200 import PackBitsTensor, _native, ops


class _Rows:
    """What ops asks of packed rows on the GPU."""
    is_cuda, dtype, device = True, torch.int32, "cpu"

    def __init__(self, rows, words):
        self.shape = (rows, words)

    def dim(self):
        return 2

    def is_contiguous(self):
        return True

    def data_ptr(self):
        return 1 << 20

    def get_device(self):
        return 0


@pytest.fixture
def lib(monkeypatch):
    from difflogic_b200 import build
    build.build()
    lib = _native.lib()
    monkeypatch.setattr(_native, "on_device", lambda t: _native._ALREADY_THERE)
    monkeypatch.setattr(_native, "stream_of", lambda t: 0)
    asked = []

    def count(x, out, n, words, pad_len, k, bits, stream):      # the library's own check, without its launch
        asked.append((words, bits))
        return _native.DL_OK if 0 <= pad_len < bits else lib.dl_groupbitsum(x, out, n, words, pad_len, k, bits, stream)
    monkeypatch.setattr(_native, "lib", lambda: type("Lib", (), {"dl_groupbitsum": staticmethod(count),
                                                                 "dl_last_error_string": lib.dl_last_error_string})())
    return asked


@pytest.mark.parametrize("words", [4, 8, 5])
@pytest.mark.parametrize("pad_len", [32, 40, 127])
def test_pad_len_beyond_a_word(lib, words, pad_len):
    x = _Rows(10, words)
    with pytest.raises(RuntimeError, match="pad_len"):
        ops.groupbitsum(x, pad_len, 2)
    if words % 4 == 0:
        assert ops.groupbitsum(x, pad_len, 2, padded=True).shape == (words * 32 - pad_len, 2) and lib[-1] == (words // 4, 128)


@pytest.mark.parametrize("pad_len", [-1, 32, 100])
def test_packed_tensor(pad_len):
    p = PackBitsTensor.from_packed(torch.zeros(10, 4, dtype=torch.int32), pad_len)
    with pytest.raises(RuntimeError, match="pad_len"):
        p.group_sum(2)
