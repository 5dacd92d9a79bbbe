"""64-wide backward on both sides of the rules that deal heads to CTAs whole or in units: against the oracle, the heads of both kernels on their own."""
import pytest
import torch

from llmc_b200 import _lib
from llmc_b200.ops import kernels as KN
from llmc_b200.ops import reference as R

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("B,T,NH", [
    (1, 256, 148), (1, 130, 149), (3, 300, 99),              # two and three tiles: whole
    (2, 300, 37), (1, 384, 75), (1, 257, 1),                 # three tiles of heads whose units a CTA has one of: split; of one head more: whole
    (2, 400, 96), (1, 512, 70), (1, 600, 190),               # four, five: whole beside whole heads / split / one full round only: split
    (1, 640, 300), (1, 1024, 300), (4, 897, 80),             # two rounds whole, the others split
    (2, 1280, 150), (1, 1281, 300),                          # the most tiles; one more
])
def test_heads_whole_and_split(B, T, NH):
    g = torch.Generator().manual_seed(B * T + NH)
    qkv, dout = torch.randn(B, T, 3 * NH * 64, generator=g).bfloat16(), torch.randn(B, T, NH * 64, generator=g).bfloat16()
    q, d = qkv.to(DEV), dout.to(DEV)
    out, lse = torch.empty(B, T, NH * 64, dtype=torch.bfloat16, device=DEV), torch.empty(B, NH, T, device=DEV)
    KN.attention_forward(out, lse, q, B, T, NH)
    got = []
    for _ in range(2):
        buf = torch.full((B + 1, T, 3 * NH * 64), 7.0, dtype=torch.bfloat16, device=DEV)
        KN.attention_backward(buf[:B], d, q, out, lse, B, T, NH)
        got.append(buf)
    assert _lib.read_status() == 0
    assert torch.equal(*got) and (got[0][B:] == 7.0).all()
    # the oracle on a few heads: the first, the last, and those around the rounds of 148
    view = got[0][:B].view(B, T, 3, NH, 64)
    for n in {0, 1, 147, 148, 149, 295, 296, 297, B * NH // 2, B * NH - 1}:
        if n >= B * NH:
            continue
        b, h = divmod(n, NH)
        one = qkv.view(B, T, 3, NH, 64)[b:b + 1, :, :, h].reshape(1, T, 192)
        ro, rl, rd = torch.empty(1, T, 64), torch.empty(1, 1, T), torch.empty(1, T, 192)
        R.attention_forward(ro, rl, one, 1, T, 1)
        R.attention_backward(rd, dout.view(B, T, NH, 64)[b:b + 1, :, h].contiguous(), one, ro, rl, 1, T, 1)
        rd = rd.view(T, 3, 64)
        for c in range(3):
            e = view[b, :, c, h].float().cpu() - rd[:, c]
            # as for the whole gradient: P, dS, O (through delta) and the result are each rounded to bf16 once, 0.0023 together
            assert float(e.norm() / rd[:, c].norm()) < 5e-3, (n, c)
            # and no tile of 128 rows is off on its own (a missing or doubled contribution is of the size of the tile's gradient)
            for t in range(0, T, 128):
                assert float(e[t:t + 128].norm()) < 0.02 * float(rd[t:t + 128, c].norm()) + 1e-3, (n, c, t)
