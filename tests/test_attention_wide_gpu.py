"""Attention kernels for head sizes above 64 at the sizes where their tiles, item walks and channel padding can go wrong, against the
fp32 restatement: a single ragged tile, odd and even numbers of query tiles, several items per CTA (more items than SMs), every
number of 16-channel steps."""
import pytest
import torch

from llmc_b200.ops import kernels as KN
from llmc_b200.ops import reference as R

pytestmark = pytest.mark.gpu
DEV = "cuda"

SHAPES = [(1, 1, 1, 72), (2, 7, 3, 128), (1, 129, 2, 88), (1, 640, 2, 104), (2, 513, 2, 128), (4, 300, 40, 80), (1, 130, 160, 120), (1, 1100, 20, 96)]


def inputs(B, T, NH, hs):
    g = torch.Generator().manual_seed(B + T + NH + hs)
    qkv = torch.randn(B, T, 3 * NH * hs, generator=g).bfloat16()
    return qkv, (torch.randn(B, T, NH * hs, generator=g) * 0.5).bfloat16()


def close(got, want, atol, rtol):
    got, want = got.float().cpu(), want.float()
    assert not ((got - want).abs() > atol + rtol * want.abs()).any(), float((got - want).abs().max())


@pytest.mark.parametrize("B,T,NH,hs", SHAPES)
def test_forward(B, T, NH, hs):
    qkv, _ = inputs(B, T, NH, hs)
    buf = torch.full((B * T + 4, NH * hs), 7.0, dtype=torch.bfloat16, device=DEV)      # rows past the end must stay untouched
    lse = torch.empty(B, NH, T, device=DEV)
    KN.attention_forward(buf[:B * T], lse, qkv.to(DEV), B, T, NH)
    ro, rl = torch.empty(B, T, NH * hs), torch.empty(B, NH, T)
    R.attention_forward(ro, rl, qkv, B, T, NH)
    close(lse, rl, 1e-3, 1e-3)
    close(buf[:B * T].view(B, T, -1), ro, 2e-2, 2e-2)          # P and the output are rounded to bf16: 2^-8 of values up to 4
    assert (buf[B * T:] == 7.0).all()


@pytest.mark.parametrize("B,T,NH,hs", SHAPES)
def test_backward(B, T, NH, hs):
    qkv, dout = inputs(B, T, NH, hs)
    ro, rl, rd = torch.empty(B, T, NH * hs), torch.empty(B, NH, T), torch.empty(B, T, 3 * NH * hs)
    R.attention_forward(ro, rl, qkv, B, T, NH)
    R.attention_backward(rd, dout, qkv, ro, rl, B, T, NH)
    got = []
    for _ in range(2):
        buf = torch.full((B * T + 4, 3 * NH * hs), 7.0, dtype=torch.bfloat16, device=DEV)
        KN.attention_backward(buf[:B * T], dout.to(DEV), qkv.to(DEV), ro.bfloat16().to(DEV), rl.to(DEV), B, T, NH)
        assert (buf[B * T:] == 7.0).all()
        got.append(buf[:B * T])
    assert torch.equal(got[0], got[1])
    # delta uses the bf16 output: its rounding (2^-9 of |O| |dO| over hs channels) times P stays below 2e-2 beside the bf16 results
    close(got[0].view(B, T, -1), rd, 4e-2, 3e-2)


@pytest.mark.parametrize("HS", [80, 128])
def test_the_largest_probability_of_a_row_is_exact(HS):
    """Rows whose largest score (4 to 5.5 above an earlier key's) comes with their second key tile and makes up nearly all of the sum: with the
    probability of that key exactly 1, the error is little more than that of rounding the result to bf16."""
    B, T, NH, lo = 1, 256, 2, 128
    g = torch.Generator().manual_seed(HS)
    q, k = torch.zeros(B, T, NH, HS), torch.zeros(B, T, NH, HS)
    v = torch.randn(B, T, NH, HS, generator=g)
    q[:, lo:, :, 0] = torch.linspace(4.0, 5.5, T - lo)[:, None] * HS ** 0.5
    q[..., 1] = HS ** 0.5
    k[..., 1] = -20.0
    k[:, 0, :, 1] = k[:, lo, :, 1] = 0.0
    k[:, lo, :, 0] = 1.0
    qkv = torch.stack([q, k, v], 2).bfloat16()
    qd, kd, vd = qkv.double().unbind(2)
    s = (torch.einsum("bthd,bshd->bhts", qd, kd) / HS ** 0.5).masked_fill(torch.ones(T, T, dtype=torch.bool).triu(1), -float("inf"))
    exact = torch.einsum("bhts,bshd->bthd", torch.softmax(s, -1), vd)[:, lo:]
    out = torch.empty(B, T, NH * HS, dtype=torch.bfloat16, device="cuda")
    lse = torch.empty(B, NH, T, device="cuda")
    KN.attention_forward(out, lse, qkv.view(B, T, 3 * NH * HS).cuda(), B, T, NH)
    err = (out.cpu().view(B, T, NH, HS)[:, lo:].double() - exact).norm()
    assert err < 1.1 * (exact.bfloat16().double() - exact).norm()


@pytest.mark.parametrize("T,HS", [(100, 80), (333, 128)])
def test_backward_with_a_key_of_score_minus_infinity(T, HS):
    """A key that no query gives any weight: the gradients of keys and values do not depend on whether its scores are -inf or very negative, also
    where the last query tile is ragged."""
    B, NH, at = 2, 2, 40
    g = torch.Generator().manual_seed(T)
    qkv = torch.randn(B, T, 3, NH, HS, generator=g)
    qkv[:, :, 0, :, 0] = qkv[:, :, 0, :, 0].abs() + 0.5
    dout = torch.randn(B, T, NH * HS, generator=g).bfloat16().cuda()
    grads = []
    for low in (-1e30, -float("inf")):
        qkv[:, at, 1, :, 0] = low
        x = qkv.bfloat16().view(B, T, 3 * NH * HS).cuda()
        out, lse, dqkv = torch.empty_like(dout), torch.empty(B, NH, T, device=DEV), torch.empty_like(x)
        KN.attention_forward(out, lse, x, B, T, NH)
        KN.attention_backward(dqkv, dout, x, out, lse, B, T, NH)
        assert out.isfinite().all() and lse.isfinite().all()
        grads.append(dqkv.view(B, T, 3, NH, HS)[:, :, 1:].clone())
    assert grads[1].isfinite().all() and torch.equal(*grads)
