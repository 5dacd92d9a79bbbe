"""What the decoding entry points decide before anything is launched: positions that they refuse, the depth of the attention kernel's ring."""
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


# either side of each line: two stages for the 128-wide fused step in clusters of long slices, about two CTAs on each of 148 SMs
@pytest.mark.parametrize("B,Tmax,NKV,HS,rope,stages", [
    (32, 2048, 8, 128, 1, 2), (32, 2048, 8, 128, 0, 3), (32, 2048, 8, 64, 1, 3), (32, 1024, 8, 128, 1, 2), (32, 960, 8, 128, 1, 3), (27, 2048, 8, 128, 1, 3),
    (28, 2048, 8, 128, 1, 2), (37, 2048, 8, 128, 1, 2), (38, 2048, 8, 128, 1, 3), (64, 2048, 8, 128, 1, 3), (8, 8192, 8, 128, 1, 2), (8, 2048, 8, 128, 1, 3),
    (1, 16384, 8, 128, 1, 3), (4, 16384, 8, 128, 1, 3)])
def test_ring(B, Tmax, NKV, HS, rope, stages):
    assert _lib.cuda().llmc_cached_attention_stages(B, Tmax, NKV, HS, rope) == stages
