"""64-wide heads at the sizes where their sequences of tiles change: one and an odd number of tiles, ragged lengths, more heads than CTAs."""
import pytest
import torch

from llmc_b200 import _lib
from llmc_b200.ops import kernels as KN
from llmc_b200.ops import reference as R

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("B,T,NH", [(2, 100, 3), (1, 129, 2), (25, 257, 6), (13, 300, 12), (4, 640, 38), (1, 2048, 5), (150, 200, 1),
                                    # one tile: every number of 16-query groups, fewer and more heads than twice the CTAs (a single token has dQ = dK = 0, of which
                                    # a relative error says nothing)
                                    (3, 5, 2), (2, 16, 3), (3, 17, 2), (30, 32, 12), (2, 33, 5), (30, 64, 12), (2, 65, 3), (30, 65, 12), (30, 96, 12), (30, 97, 12), (2, 128, 5)])
def test_forward_and_backward(B, T, NH):
    g = torch.Generator().manual_seed(B * T + NH)
    qkv, dout = torch.randn(B, T, 3 * NH * 64, generator=g).bfloat16(), torch.randn(B, T, NH * 64, generator=g).bfloat16()
    ro, rl, rd = torch.empty(B, T, NH * 64), torch.empty(B, NH, T), torch.empty(B, T, 3 * NH * 64)
    R.attention_forward(ro, rl, qkv, B, T, NH)
    R.attention_backward(rd, dout, qkv, ro, rl, B, T, NH)
    rel = lambda a, r: float((a.float().cpu() - r).norm() / r.norm())
    got = []
    for _ in range(2):
        out = torch.full((B + 1, T, NH * 64), 7.0, dtype=torch.bfloat16, device=DEV)
        lse = torch.empty(B, NH, T, device=DEV)
        buf = torch.full((B + 1, T, 3 * NH * 64), 7.0, dtype=torch.bfloat16, device=DEV)
        KN.attention_forward(out[:B], lse, qkv.to(DEV), B, T, NH)
        KN.attention_backward(buf[:B], dout.to(DEV), qkv.to(DEV), out[:B], lse, B, T, NH)
        got.append((out, lse, buf))
    assert _lib.read_status() == 0
    assert all(torch.equal(x, y) for x, y in zip(*got))
    out, lse, buf = got[0]
    assert (out[B:] == 7.0).all() and (buf[B:] == 7.0).all()
    # P, dS, O (through delta) and the result are each rounded to bf16 once, 2^-9 / sqrt(3) = 0.0011 in the mean square: 0.0023 together
    assert rel(out[:B], ro) < 4e-3 and float((lse.cpu() - rl).abs().max()) < 1e-4
    for c in range(3):
        s = slice(c * NH * 64, (c + 1) * NH * 64)
        assert rel(buf[:B, :, s], rd[..., s]) < 5e-3, c


@pytest.mark.parametrize("B,T,NH,ramp", [
    # both slots of a block on one query tile: two key tiles, ragged and whole last ones, as many query tiles as three per SM (148 SMs); then more
    (1, 66, 2, 0), (1, 191, 3, 0), (1, 192, 3, 0), (1, 193, 3, 0), (2, 450, 7, 0), (37, 200, 6, 0), (223, 129, 1, 0),
    # scores that grow along the keys: the reference maximum moves in most tiles
    (1, 900, 3, 1), (40, 300, 6, 1)])
def test_forward_slots(B, T, NH, ramp):
    g = torch.Generator().manual_seed(B + T + NH)
    qkv = torch.randn(B, T, 3 * NH * 64, generator=g)
    if ramp:
        q, k = qkv[..., :NH * 64], qkv[..., NH * 64:2 * NH * 64]
        q.copy_(q.abs())
        k.copy_(k.abs() * torch.linspace(0.1, 4.0, T).view(1, T, 1))
    qkv = qkv.bfloat16()
    ro, rl = torch.empty(B, T, NH * 64), torch.empty(B, NH, T)
    R.attention_forward(ro, rl, qkv, B, T, NH)
    out = torch.full((B + 1, T, NH * 64), 7.0, dtype=torch.bfloat16, device=DEV)
    lse = torch.empty(B, NH, T, device=DEV)
    KN.attention_forward(out[:B], lse, qkv.to(DEV), B, T, NH)
    assert _lib.read_status() == 0 and (out[B:] == 7.0).all()
    # P and O rounded to bf16 once each: 0.0016 together; LSE of up to 200 in fp32
    assert float((out[:B].float().cpu() - ro).norm() / ro.norm()) < 4e-3
    assert float((lse.cpu() - rl).abs().max()) < 1e-4 + 2e-6 * float(rl.abs().max())


@pytest.mark.parametrize("B", [1, 40])                # one / two query tiles to a CTA
def test_a_nan_key_reaches_its_queries(B):
    """Head h has a NaN in key 3 h: every place of a group of exponentials, whichever unit takes it."""
    T, NH = 130, 24
    qkv = torch.randn(B, T, 3, NH, 64, generator=torch.Generator().manual_seed(B)).bfloat16()
    for h in range(NH):
        qkv[:, 3 * h, 1, h, 5] = float("nan")
    out, lse = torch.empty(B, T, NH * 64, dtype=torch.bfloat16, device=DEV), torch.empty(B, NH, T, device=DEV)
    KN.attention_forward(out, lse, qkv.view(B, T, -1).to(DEV), B, T, NH)
    assert _lib.read_status() == 0
    seen = torch.arange(T)[None, :] >= 3 * torch.arange(NH)[:, None]                     # (NH, T)
    assert torch.equal(lse.isnan().cpu(), seen.expand(B, -1, -1))
    assert torch.equal(out.view(B, T, NH, 64).isnan().cpu(), seen.t()[None, :, :, None].expand(B, -1, -1, 64))


# one query tile to a slot (12 x 700 x 16 heads are more than three tiles per SM, 1 x 777 x 8 are not: both slots on one), ragged and whole tiles
@pytest.mark.parametrize("B,T,NH", [(12, 700, 16), (24, 129, 16), (16, 300, 12), (8, 1024, 16), (1, 777, 8)])
def test_error_is_that_of_probabilities_rounded_once(B, T, NH):
    """O in 64 bits with each row's probabilities relative to its maximum over the first 128 keys and rounded to bf16, the result rounded once more: the kernel is
    no further from the exact O than that.  Both round the same 10^6 to 10^7 values, so that their errors differ by far less than the 0.2 % allowed
    here; a reference that is the maximum of 64 keys makes 0.4 to 0.9 % more."""
    g = torch.Generator(device=DEV).manual_seed(B * T)
    qkv = torch.randn(B, T, 3 * NH * 64, generator=g, device=DEV).bfloat16()
    out, lse = torch.empty(B, T, NH * 64, dtype=torch.bfloat16, device=DEV), torch.empty(B, NH, T, device=DEV)
    KN.attention_forward(out, lse, qkv, B, T, NH)
    err = rounded = norm = 0.0
    hidden = torch.ones(T, T, dtype=torch.bool, device=DEV).triu(1)
    for b in range(B):
        q, k, v = qkv[b].view(T, 3, NH, 64).permute(1, 2, 0, 3).double()
        s = (q @ k.transpose(1, 2) / 8).masked_fill(hidden, -torch.inf)
        p = torch.exp(s - s[..., :128].amax(-1, keepdim=True))
        exact = p @ v / p.sum(-1, keepdim=True)
        once = (p.bfloat16().double() @ v / p.sum(-1, keepdim=True)).bfloat16().double()
        err += float((out[b].view(T, NH, 64).transpose(0, 1).double() - exact).square().sum())
        rounded += float((once - exact).square().sum())
        norm += float(exact.square().sum())
    assert _lib.read_status() == 0
    assert err ** 0.5 < 1.002 * rounded ** 0.5, ((err / norm) ** 0.5, (rounded / norm) ** 0.5)

# keys 0 .. 63 (of some heads 0 .. 127: whole tiles that a row sees nothing in) with scores that overflow
@pytest.mark.parametrize("B", [1, 40])
def test_infinite_scores_in_the_first_tiles(B):
    T, NH = 330, 24
    qkv = torch.randn(B, T, 3, NH, 64, generator=torch.Generator().manual_seed(B)).bfloat16()
    qkv[:, :, 0, :, 7], qkv[:, :, 1, :, 7] = 1e20, 0.0
    first = torch.tensor([64, 128, 40, 100, 200, 0]).repeat(NH // 6)       # keys of a head that score -inf
    for h in range(NH):
        qkv[:, :first[h], 1, h, 7] = -1e20
    out, lse = torch.empty(B, T, NH * 64, dtype=torch.bfloat16, device=DEV), torch.empty(B, NH, T, device=DEV)
    KN.attention_forward(out, lse, qkv.view(B, T, -1).to(DEV), B, T, NH)
    assert _lib.read_status() == 0
    q, k, v = qkv.float().permute(2, 0, 3, 1, 4)
    keys = torch.arange(T)
    hidden = (keys[None, :] > keys[:, None])[None] | (keys[None, None, :] < first[:, None, None])       # (NH, T, T)
    q[..., 7] = k[..., 7] = 0.0
    s = (q @ k.transpose(2, 3) / 8).masked_fill(hidden, -torch.inf)
    # a row all of whose scores are -inf has no softmax
    seen = keys[None, :] >= first[:, None]
    ref = torch.softmax(s, -1) @ v
    got = out.view(B, T, NH, 64).transpose(1, 2).float().cpu()
    assert torch.equal(got.isnan().any(-1), ~seen.expand(B, -1, -1)) and torch.equal(got.isnan().all(-1), ~seen.expand(B, -1, -1))
    assert torch.equal(lse.isnan().cpu(), ~seen.expand(B, -1, -1))
    got, ref = got[seen.expand(B, -1, -1)], ref[seen.expand(B, -1, -1)]
    assert float((got - ref).norm() / ref.norm()) < 4e-3                   # P and O rounded to bf16 once each
    assert torch.allclose(lse.cpu()[seen.expand(B, -1, -1)], torch.logsumexp(s, -1)[seen.expand(B, -1, -1)], atol=1e-4)
