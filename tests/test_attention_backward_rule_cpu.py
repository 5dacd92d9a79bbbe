"""How the 64-wide backward deals its heads on 148 SMs: whole (two launches), whole and split (four), all split (three), one tile (one)."""
import pytest

from llmc_b200 import _lib


@pytest.mark.parametrize("B,T,NH,launches", [
    (5, 128, 12, 1), (1, 129, 1, 2), (4, 256, 12, 2), (40, 256, 12, 2),                    # two tiles: nothing gets shorter by splitting
    (1, 300, 12, 3), (2, 384, 37, 3), (1, 384, 75, 2), (12, 384, 12, 2), (16, 300, 12, 2),  # three: as long as no CTA has two units
    (4, 512, 12, 3), (8, 512, 12, 2), (8, 640, 12, 2), (4, 640, 12, 3),
    (13, 1024, 12, 3), (37, 1024, 12, 2), (64, 1024, 12, 4), (32, 1280, 12, 4), (37, 1280, 12, 2), (37, 1281, 12, 3)])
def test_launches(B, T, NH, launches):
    assert _lib.cuda().llmc_attention_bwd_launches(B, T, NH, 64) == launches
