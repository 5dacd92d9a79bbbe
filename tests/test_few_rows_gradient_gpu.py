"""Input gradients of some hundred rows through the split-K kernel (csrc/stream_gemm.cu): row tiles of 48 to 128 rows and, for deep products, of up to 256, two, four and eight slices of K, ragged
rows, columns and depths, and either side of the line where the dispatch takes it."""
import pytest
import torch

from llmc_b200 import _lib
from llmc_b200.ops import kernels as KN

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("M,N,K", [(129, 8, 8), (130, 136, 200), (256, 768, 768), (257, 264, 392), (300, 768, 2304), (400, 2048, 776), (256, 1000, 3080), (1024, 768, 3072), (384, 768, 6152), (200, 1600, 8200),
                                   (500, 2056, 768), (1000, 2048, 768)])
def test_product(M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    dy, w = torch.randn(M, K, generator=g).bfloat16().to(DEV), (torch.randn(K, N, generator=g) * 0.05).bfloat16().to(DEV)
    want = dy.double() @ w.double()
    got = []
    for _ in range(2):
        out = torch.full((M + 3, N), 7.0, dtype=torch.bfloat16, device=DEV)
        assert _lib.cuda().llmc_stream_gemm(KN._p(out), KN._p(dy), KN._p(w), None, M, N, K, K, N, N, 1, KN._stream()) == 0
        got.append(out)
    assert torch.equal(*got) and (got[0][M:] == 7.0).all() and _lib.read_status() == 0
    # one rounding to bf16 (half a unit of 8 significant bits: 2^-8 of the value at most) of a sum in fp32, whose own error is below K * 2^-24 times the
    # sum of the magnitudes
    bound = 2 ** -8 * want.abs() + K * 2 ** -24 * (dy.double().abs() @ w.double().abs()) + 1e-6
    assert not ((got[0][:M].double() - want).abs() > bound).any()


# depth, rows and columns on either side of each line
@pytest.mark.parametrize("M,N,K,taken", [(256, 768, 768, True), (256, 768, 760, False), (1024, 1024, 2048, True), (1024, 1024, 2040, False), (1025, 1024, 3064, False),
                                         (129, 4096, 2048, True), (129, 4224, 3064, False)])
def test_dispatch(M, N, K, taken):
    assert KN._few_rows(M, N, K, KN.MODE_STORE, True, torch.device(DEV, 0)) == taken
    assert not KN._few_rows(M, N, K, KN.MODE_DGELU, True, torch.device(DEV, 0))
