"""Positions that the decoding entry points refuse before anything is launched."""
import pytest

from llmc_b200 import _lib

LARGEST = 2 ** 31 - 1


@pytest.mark.parametrize("start,Tq,freqs_len,rc", [(40, 1, 64, -2), (-1, 1, 64, -2), (LARGEST, 1, 64, -2), (LARGEST - 3, 8, 64, -2), (30, 1, 30, -4), (0, 8, 4, -4)])
def test_positions(start, Tq, freqs_len, rc):
    lib = _lib.cuda()
    one = 4096                                   # an address: nothing is read
    assert lib.llmc_rope_cache(one, one, one, one, one, freqs_len, 1, Tq, 40, start, 2, 1, 64, None, None) == rc
    assert lib.llmc_cached_attention_rope(one, one, one, freqs_len, one, one, 1, Tq, 40, start, 2, 1, 64, None, None, 0, None) == rc
    if rc == -2:
        assert lib.llmc_cached_attention(one, one, one, one, 1, Tq, 40, start, 2, 1, 64, None, None, None) == rc
