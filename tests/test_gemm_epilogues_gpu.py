"""The epilogues of the two-SM GEMM that move a second tensor (GELU, dGELU, accumulation without split-K): ragged tiles in both directions
and more tiles than CTA pairs, so that a warp's staging buffer and prefetched piece are reused from tile to tile."""
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


@pytest.mark.parametrize("M,N,K", [(5000, 1032, 72), (300, 72, 200), (20000, 264, 64)])
def test_gelu_and_its_gradient(M, N, K, monkeypatch):
    monkeypatch.setattr(KN, "TWO_SM_MIN_TILES", 1)
    x, w, b, dy, w2 = rnd(M, K), rnd(N, K, scale=0.05, seed=1), rnd(N, seed=2), rnd(M, K, seed=3), rnd(K, N, scale=0.05, seed=4)
    out = torch.full((M + 2, N), 7.0, dtype=torch.bfloat16, device=DEV)
    pre = torch.full((M + 2, N), 7.0, dtype=torch.bfloat16, device=DEV)
    KN.matmul_forward(out[:M], x.to(DEV), w.to(DEV), b.to(DEV), pre_gelu=pre[:M])
    ref, refpre = torch.empty(M, N), torch.empty(M, N)
    R.matmul_forward(ref, x, w, b, pre_gelu=refpre)
    close(pre[:M], refpre, 2e-2, 1e-2)
    close(out[:M], ref, 2e-2, 1e-2)
    again = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    KN.gelu_forward(again, pre[:M])
    assert torch.equal(again, out[:M])                         # a recomputed activation has the bits of the stored one
    KN.matmul_dgrad(out[:M], dy.to(DEV), w2.to(DEV), pre_gelu=pre[:M])
    R.matmul_dgrad(ref, dy, w2, pre_gelu=pre[:M].cpu())
    close(out[:M], ref, 3e-2, 1e-2)
    assert (out[M:] == 7.0).all() and (pre[M:] == 7.0).all()


@pytest.mark.parametrize("rows,OC,C", [(512, 2000, 1544), (72, 5000, 1032), (256, 3072, 768)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_weight_gradient_without_split(rows, OC, C, accumulate):
    dy, x, dw0 = rnd(rows, OC, scale=0.1), rnd(rows, C), rnd(OC, C, seed=5)
    buf = torch.full((OC + 2, C), 7.0, dtype=torch.bfloat16, device=DEV)
    buf[:OC] = dw0.to(DEV)
    KN.matmul_wgrad(buf[:OC], dy.to(DEV), x.to(DEV), accumulate=accumulate)
    ref = dw0.float().clone()
    R.matmul_wgrad(ref, dy, x, accumulate=accumulate)
    close(buf[:OC], ref, 5e-2, 1.5e-2)
    assert (buf[OC:] == 7.0).all()


@pytest.mark.parametrize("two_sm", [False, True])
def test_gelu_gradient_of_large_inputs(two_sm, monkeypatch):
    """Far from zero the derivative is exactly 0 or 1, up to the largest x whose square is finite: stand-alone and in both GEMM epilogues."""
    monkeypatch.setattr(KN, "TWO_SM_MIN_TILES", 1 if two_sm else 0)
    x = torch.tensor([s * m * 10.0 ** e for e in range(1, 19) for m in (1.0, 3.0) for s in (1.0, -1.0)]).bfloat16()
    want = (x > 0).float()
    d = torch.ones_like(x).to(DEV)
    KN.gelu_backward_inplace(d, x.to(DEV))
    assert torch.equal(d.float().cpu(), want)
    M, N = 256, x.numel()
    pre, dy, w = x.expand(M, N).contiguous(), torch.ones(M, 8), torch.full((8, N), 0.125)
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    KN.matmul_dgrad(out, dy.bfloat16().to(DEV), w.bfloat16().to(DEV), pre_gelu=pre.to(DEV))
    assert torch.equal(out.float().cpu(), want.expand(M, N))


@pytest.mark.parametrize("two_sm", [False, True])
@pytest.mark.parametrize("M,N,K", [(640, 152, 96), (942, 184, 24), (1541, 152, 8), (952, 440, 1112), (1950, 1944, 304), (300, 1600, 64), (20000, 136, 16), (3000, 8, 64)])
def test_last_columns_of_a_ragged_output(two_sm, M, N, K, monkeypatch):
    """Outputs that end early in a tile: the empty column chunks behind the last one share its staging buffers.  Many fresh outputs, since a
    buffer that is reused too early shows only when its store is slow."""
    monkeypatch.setattr(KN, "TWO_SM_MIN_TILES", 1 if two_sm else 0)
    x, w = rnd(M, K).to(DEV), rnd(N, K, scale=K ** -0.5, seed=1).to(DEV)
    wt = w.t().contiguous()
    want = x.float() @ w.float().t()
    for _ in range(20):
        for product, weight in ((KN.matmul_forward, w), (KN.matmul_dgrad, wt)):
            out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
            product(out, x, weight)
            assert not ((out.float() - want).abs() > 2e-2 + 1e-2 * want.abs()).any()
