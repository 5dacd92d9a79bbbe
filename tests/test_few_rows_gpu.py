"""Kernels of decoding steps and short prompts at the edges of their tiles and splits, against the fp32 restatement."""
import pytest
import torch

from llmc_b200.ops import kernels as KN
from llmc_b200.ops import reference as R

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rnd(*shape, scale=1.0, seed=0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g) * scale).bfloat16()


def close(got, want, atol, rtol):
    got, want = got.float().cpu(), want.float()
    assert not ((got - want).abs() > atol + rtol * want.abs()).any(), float((got - want).abs().max())


# one row to a full tile; rows around the multiples of 16; ragged and tiny N; one K block, a K tail, K blocks that do not divide by the split
@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (9, 130, 200), (16, 2048, 2048), (17, 999, 4096), (33, 6144, 1000), (64, 64, 72), (100, 40000, 136),
                                   (127, 256, 7168), (128, 3072, 2048)])
@pytest.mark.parametrize("bias", [False, True])
def test_forward_product_of_few_rows(M, N, K, bias):
    x, w, b = rnd(M, K), rnd(N, K, scale=0.05, seed=1), rnd(N, seed=2) if bias else None
    # 16 rows of canaries below the output
    buf = torch.full((M + 16, N), 7.0, dtype=torch.bfloat16, device=DEV)
    KN.matmul_forward(buf[:M], x.to(DEV), w.to(DEV), b.to(DEV) if bias else None)
    ref = torch.empty(M, N)
    R.matmul_forward(ref, x, w, b)
    close(buf[:M], ref, 2e-2, 1e-2)
    assert (buf[M:] == 7.0).all()
    again = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    KN.matmul_forward(again, x.to(DEV), w.to(DEV), b.to(DEV) if bias else None)
    assert torch.equal(again, buf[:M])


@pytest.mark.parametrize("M,H,K", [(1, 64, 64), (4, 7168, 2048), (31, 192, 520), (128, 1024, 256)])
def test_swiglu_product(M, H, K):
    x, w = rnd(M, K), rnd(2 * H, K, scale=0.05, seed=1)
    h = torch.full((M + 2, H), 7.0, dtype=torch.bfloat16, device=DEV)
    KN.matmul_swiglu(h[:M], x.to(DEV), w.to(DEV))
    ref = torch.empty(M, H)
    R.matmul_swiglu(ref, x, w)
    close(h[:M], ref, 3e-2, 1e-2)
    assert (h[M:] == 7.0).all()


# position 0, a partial first tile, several tiles per warp, one slice, a cluster of slices, more slices than a cluster holds
@pytest.mark.parametrize("B,Tq,start,Tmax,NH,NKV,HS", [(1, 1, 0, 8, 2, 2, 64), (2, 1, 14, 192, 8, 2, 64), (1, 2, 126, 1024, 8, 2, 128), (3, 1, 1500, 1600, 4, 1, 128),
                                                       (1, 1, 9000, 9100, 2, 1, 64), (40, 1, 77, 300, 16, 8, 64), (1, 8, 250, 600, 2, 2, 128)])
def test_cached_attention(B, Tq, start, Tmax, NH, NKV, HS):
    q, kc, vc = rnd(B * Tq, NH * HS), rnd(B, Tmax, NKV, HS, seed=1), rnd(B, Tmax, NKV, HS, seed=2)
    kc[:, start + Tq:] = float("nan")                          # positions that no query may see
    vc[:, start + Tq:] = float("nan")
    ref = torch.empty(B * Tq, NH * HS)
    R.cached_attention(ref, q, kc, vc, Tq, start, NH, NKV)
    out = torch.empty(B * Tq, NH * HS, dtype=torch.bfloat16, device=DEV)
    KN.cached_attention(out, q.to(DEV), kc.to(DEV), vc.to(DEV), Tq, start, NH, NKV)
    close(out, ref, 4e-3, 8e-3)                                # one rounding to bf16 (2^-9)


@pytest.mark.parametrize("HS,start,Tmax", [(64, 159, 192), (128, 999, 1000)])
def test_cached_attention_keeps_fp32_probabilities(HS, start, Tmax):
    """Values chosen so that the weighted sum cancels to about 2^-18 of its terms.  Probabilities in fp32 (the exponential and its argument
    are good to 2^-22) leave an error of 2^-8 of the result, next to its rounding to bf16 (2^-9); with 16 bits it would be 2^-5 and 2^-4."""
    B, NH = 4, 8
    g = torch.Generator().manual_seed(start)
    q, kc = rnd(B, NH * HS), rnd(B, Tmax, NH, HS, seed=1)
    n = start + 1
    p = torch.softmax(torch.einsum("bhd,bshd->bhs", q.view(B, NH, HS).double(), kc[:, :n].double()) / HS ** 0.5, -1)
    v = torch.randn(B, NH, n, HS, generator=g).bfloat16().double()
    want = torch.randn(B, NH, HS, generator=g).double() * 2.0 ** -18
    top = p.topk(2, -1)
    for i in range(2):                                         # the two largest probabilities take up what is left
        at = top.indices[..., i, None, None].expand(B, NH, 1, HS)
        if i == 0:
            v.scatter_(2, top.indices[..., None].expand(B, NH, 2, HS), 0.0)
        left = want - torch.einsum("bhs,bhsd->bhd", p, v)
        v.scatter_(2, at, (left / top.values[..., i, None]).bfloat16().double()[:, :, None])
    exact = torch.einsum("bhs,bhsd->bhd", p, v).view(B, NH * HS)
    vc = torch.zeros(B, Tmax, NH, HS, dtype=torch.bfloat16)
    vc[:, :n] = v.transpose(1, 2).bfloat16()
    out = torch.empty(B, NH * HS, dtype=torch.bfloat16, device=DEV)
    KN.cached_attention(out, q.to(DEV), kc.to(DEV), vc.to(DEV), 1, start, NH, NH)
    err = (out.cpu().double() - exact).norm() / exact.norm()
    assert err < 2.0 ** -6, float(err)


@pytest.mark.parametrize("start,Tmax", [(0, 8), (14, 192), (77, 1024), (2000, 2100)])
@pytest.mark.parametrize("HS", [64, 128])
def test_cached_attention_with_infinite_values(HS, start, Tmax):
    """An infinite value gives that infinity in its channel whatever its probability (also one with a single bit), and nothing elsewhere."""
    B, NH, NKV = 2, 8, 2
    q, kc, vc = rnd(B, NH * HS), rnd(B, Tmax, NKV, HS, seed=1), rnd(B, Tmax, NKV, HS, seed=2)
    kc[0] = 0.0                                                # equal scores: every probability of a tile is exactly 1
    vc[:, start, :, 3], vc[:, start // 2, :, 9] = float("inf"), float("-inf")
    vc[:, start + 1:] = float("nan")
    ref = torch.empty(B, NH * HS)
    R.cached_attention(ref, q, kc, vc, 1, start, NH, NKV)
    assert ref.isinf().sum() == 2 * B * NH and not ref.isnan().any()
    out = torch.empty(B, NH * HS, dtype=torch.bfloat16, device=DEV)
    KN.cached_attention(out, q.to(DEV), kc.to(DEV), vc.to(DEV), 1, start, NH, NKV)
    got, inf = out.float().cpu(), ref.isinf()
    assert torch.equal(got[inf], ref[inf])
    close(got[~inf], ref[~inf], 4e-3, 8e-3)


@pytest.mark.parametrize("N,C", [(1, 8), (3, 264), (5, 2048), (1024, 512), (1025, 512), (4, 2056), (2, 8192), (2, 16384), (2, 16392)])
def test_rmsnorm_forward(N, C):
    a, b, w = rnd(N, C), rnd(N, C, seed=3), rnd(C) + 1.0
    res, out = torch.empty(N, C, dtype=torch.bfloat16, device=DEV), torch.empty(N, C, dtype=torch.bfloat16, device=DEV)
    rstd = torch.empty(N, device=DEV)
    KN.rmsnorm_fused_residual_forward(res, out, rstd, a.to(DEV), b.to(DEV), w.to(DEV))
    rres, ro, rr = torch.empty(N, C, dtype=torch.bfloat16), torch.empty(N, C), torch.empty(N)
    R.rmsnorm_fused_residual_forward(rres, ro, rr, a, b, w)
    assert torch.equal(res.cpu(), rres)
    close(rstd, rr, 0, 1e-5)
    close(out, ro, 1e-2, 1.2e-2)                               # two roundings to bf16
    KN.rmsnorm_forward(out, rstd, res, w.to(DEV))
    close(out, ro, 1e-2, 1.2e-2)
