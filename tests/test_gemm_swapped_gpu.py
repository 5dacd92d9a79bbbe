"""The two-SM GEMM with swapped operand roles (csrc/gemm2t.cu): every number of activation rows per tile that changes its layout, ragged rows, columns and
depths, and the SwiGLU form."""
import pytest
import torch

from llmc_b200 import _lib
from llmc_b200.ops import kernels as KN

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rnd(*shape, scale=1.0, seed=0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g) * scale).bfloat16().to(DEV)


# one rounding to bf16 (2^-9 at most) of a sum that is exact to fp32; 1e-3 for results near zero
def close(got, want, rtol=2 ** -8, atol=1e-3):
    got, want = got.float(), want.float()
    assert not ((got - want).abs() > atol + rtol * want.abs()).any(), float((got - want).abs().max())


@pytest.mark.parametrize("rows", [0, 16, 48, 112, 256])
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (130, 264, 200), (300, 1000, 72), (777, 520, 136), (2500, 72, 64)])
def test_product(rows, M, N, K):
    x, w, b = rnd(M, K), rnd(N, K, scale=0.1, seed=1), rnd(N, seed=2)
    out = torch.full((M + 3, N), 7.0, dtype=torch.bfloat16, device=DEV)
    assert _lib.cuda().llmc_gemm2t(KN._p(out), KN._p(x), KN._p(w), KN._p(b), M, N, K, K, K, N, rows, KN._stream()) == 0
    close(out[:M], (x.double() @ w.double().t() + b.double()).float())
    assert (out[M:] == 7.0).all() and _lib.read_status() == 0


@pytest.mark.parametrize("rows", [0, 16, 144, 256])
@pytest.mark.parametrize("M,H,K", [(5, 128, 64), (300, 384, 200), (900, 1024, 72)])
def test_swiglu(rows, M, H, K):
    x, w = rnd(M, K), rnd(2 * H, K, scale=0.1, seed=1)
    out = torch.full((M + 3, H), 7.0, dtype=torch.bfloat16, device=DEV)
    assert _lib.cuda().llmc_gemm2t_swiglu(KN._p(out), KN._p(x), KN._p(w), M, H, K, K, K, H, rows, KN._stream()) == 0
    u = x.double() @ w.double().t()
    close(out[:M], (u[:, :H] * torch.nn.functional.silu(u[:, H:])).float())
    assert (out[M:] == 7.0).all() and _lib.read_status() == 0


@pytest.mark.parametrize("M,K,N", [(300, 1024, 264), (777, 2048, 520), (2000, 1032, 136)])
def test_forward_products_take_it(M, K, N):
    """The launcher sends them there with the caller's own tensors: out may have more rows, the bias is added."""
    x, w, b = rnd(M, K), rnd(N, K, scale=0.05, seed=1), rnd(N, seed=2)
    out = torch.full((M + 2, N), 7.0, dtype=torch.bfloat16, device=DEV)
    assert KN._swapped(M, N, K, out.device)
    KN.matmul_forward(out, x, w, b)
    close(out[:M], (x.double() @ w.double().t() + b.double()).float())
    assert (out[M:] == 7.0).all()


@pytest.mark.parametrize("M,N,K,offset", [(500, 2052, 14336, 0), (385, 2052, 6144, 0), (2048, 1004, 6144, 0), (385, 2049, 6144, 0), (500, 2056, 6144, 4), (500, 2056, 6144, 1)])
def test_outputs_it_cannot_store(M, N, K, offset):
    """Rows that are not whole 16 bytes, or an output that does not start on a 16-byte boundary."""
    x, w, b = rnd(M, K), rnd(N, K, scale=0.05, seed=1), rnd(N, seed=2)
    flat = torch.full((M * N + 16,), 7.0, dtype=torch.bfloat16, device=DEV)
    out = flat[offset:offset + M * N].view(M, N)
    KN.matmul_forward(out, x, w, b)
    want = x.double() @ w.double().t() + b.double()
    # one rounding to bf16 of an fp32 sum whose own error is below K * 2^-24 times the sum of the magnitudes
    bound = 2 ** -8 * want.abs() + K * 2 ** -24 * (x.double().abs() @ w.double().abs().t()) + 1e-3
    assert not ((out.double() - want).abs() > bound).any()
    assert (flat[:offset] == 7.0).all() and (flat[offset + M * N:] == 7.0).all()


def test_refuses_what_it_cannot_do():
    x, w, out = rnd(32, 64), rnd(64, 64), torch.empty(32, 64, dtype=torch.bfloat16, device=DEV)
    lib, p, s = _lib.cuda(), KN._p, KN._stream()
    assert lib.llmc_gemm2t(p(out), p(x), p(w), None, 32, 64, 60, 64, 64, 64, 0, s) == -1
    assert lib.llmc_gemm2t(p(out), p(x), p(w), None, 32, 64, 64, 64, 64, 64, 24, s) == -1
    assert lib.llmc_gemm2t_swiglu(p(out), p(x), p(w), 32, 32, 64, 64, 64, 64, 0, s) == -1
