"""Both layouts of the split-K kernel for products with few tiles (csrc/stream_gemm.cu) at the edges of its tiles, splits and row tiles, against
the fp32 restatement, and the sizes at which the dispatch changes over."""
import pytest
import torch

from llmc_b200 import _lib
from llmc_b200.ops import kernels as KN
from llmc_b200.ops import reference as R

pytestmark = pytest.mark.gpu
DEV = "cuda"

# one tile row, a ragged row tile, several row tiles that M does not divide evenly into; K tails, one K block, more K than one slice
SHAPES = [(1, 64, 64), (129, 136, 200), (256, 768, 3072), (257, 264, 72), (300, 130 * 8, 1000), (777, 2048, 640), (513, 8, 4096)]


def rnd(*shape, scale=1.0, seed=0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g) * scale).bfloat16()


def close(got, want, atol, rtol):
    got, want = got.float().cpu(), want.float()
    assert not ((got - want).abs() > atol + rtol * want.abs()).any(), float((got - want).abs().max())


def product(x, w, N, w_mn=False, bias=None):
    M, K = x.shape
    buf = torch.full((M + 3, N), 7.0, dtype=torch.bfloat16, device=DEV)
    p = KN._p
    _lib.check(_lib.cuda().llmc_stream_gemm(p(buf), p(x), p(w), p(bias), M, N, K, K, w.shape[1], N, int(w_mn), KN._stream()), "llmc_stream_gemm")
    assert (buf[M:] == 7.0).all()
    return buf[:M]


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_forward(M, N, K):
    x, w, b = rnd(M, K), rnd(N, K, scale=0.05, seed=1), rnd(N, seed=2)
    ref = torch.empty(M, N)
    R.matmul_forward(ref, x, w, b)
    close(product(x.to(DEV), w.to(DEV), N, bias=b.to(DEV)), ref, 2e-2, 1e-2)


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_input_gradient(M, N, K):
    dy, w = rnd(M, K), rnd(K, N, scale=0.05, seed=1)
    ref = torch.empty(M, N)
    R.matmul_dgrad(ref, dy, w)
    close(product(dy.to(DEV), w.to(DEV), N, w_mn=True), ref, 3e-2, 1e-2)


# one size on either side of each line of the rule: rows, tiles at both depths, depth of an input gradient
@pytest.mark.parametrize("M,N,K,forward,gradient", [(64, 256, 64, True, False), (65, 128 * 297, 64, False, False), (129, 256, 64, False, False),
                                                    (128, 256, 2048, True, True), (1024, 1024, 3072, False, True), (1025, 1024, 3072, False, False),
                                                    (512, 4096, 6144, True, True), (513, 4096, 6144, False, False)])
def test_dispatch(M, N, K, forward, gradient):
    dev = torch.device(DEV, 0)
    assert KN._few_rows(M, N, K, KN.MODE_STORE, False, dev) == forward
    assert KN._few_rows(M, N, K, KN.MODE_STORE, True, dev) == gradient
    assert not KN._few_rows(M, N, K, KN.MODE_GELU, False, dev) and not KN._few_rows(M, N, K, KN.MODE_DGELU, True, dev)


# forward products cut like input gradients: row tiles that do not divide the rows, ragged columns, a K tail, one row tile and many
@pytest.mark.parametrize("M,N,K", [(129, 768, 768), (200, 130, 1000), (257, 999, 3080), (1000, 384, 1536), (300, 2048, 7168), (1024, 1024, 4096)])
def test_sliced_forward(M, N, K):
    assert KN.forward_kernel(M, N, K, torch.device(DEV, 0)) == KN.FORWARD_SLICED
    x, w, b = rnd(M, K), rnd(N, K, scale=0.05, seed=1), rnd(N, seed=2)
    buf = torch.full((M + 16, N), 7.0, dtype=torch.bfloat16, device=DEV)
    KN.matmul_forward(buf[:M], x.to(DEV), w.to(DEV), b.to(DEV))
    # against 64 bits: one rounding to bf16 (2^-9) of the sum and of nothing before it
    ref = (x.double() @ w.double().t() + b.double()).float()
    close(buf[:M], ref, 1e-3, 2.0 ** -8)
    assert (buf[M:] == 7.0).all()
