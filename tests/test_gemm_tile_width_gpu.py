"""The single-SM GEMM with tiles of 64, 128 and 256 columns: ragged rows, columns and depths, all of its epilogues."""
import ctypes

import pytest
import torch

from llmc_b200 import _lib
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


@pytest.mark.parametrize("bn", [64, 128, 256])
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (130, 72, 200), (257, 264, 64), (128, 1000, 776), (3000, 520, 72)])
@pytest.mark.parametrize("mode", ["store", "gelu", "dgrad", "dgelu", "wgrad"])
def test_tile_width(bn, M, N, K, mode):
    a, w, b, aux = rnd(M, K), rnd(N, K, scale=0.05, seed=1), rnd(N, seed=2), rnd(M, N, seed=3)
    out = torch.full((M + 2, N), 7.0, dtype=torch.bfloat16, device=DEV)
    ref, refpre = torch.empty(M, N), torch.empty(M, N)
    A, B, a_mn, b_mn, md, bias, pre = a, w, 0, 0, KN.MODE_STORE, None, None
    if mode in ("store", "gelu"):
        bias = b.to(DEV)
        md = KN.MODE_GELU if mode == "gelu" else KN.MODE_STORE
        R.matmul_forward(ref, a, w, b, pre_gelu=refpre if mode == "gelu" else None)
        pre = torch.empty(M, N, dtype=torch.bfloat16, device=DEV) if mode == "gelu" else None
    elif mode in ("dgrad", "dgelu"):
        B, b_mn = w.t().contiguous(), 1
        md = KN.MODE_DGELU if mode == "dgelu" else KN.MODE_STORE
        pre = aux.to(DEV) if mode == "dgelu" else None
        R.matmul_dgrad(ref, a, B, pre_gelu=aux if mode == "dgelu" else None)
    else:
        if M % 8:
            pytest.skip("the rows of a weight gradient are channels: multiples of 8")
        A, B, a_mn, b_mn, md = a.t().contiguous(), w.t().contiguous(), 1, 1, KN.MODE_ACCUM
        out[:M] = aux.to(DEV)
        ref.copy_(aux.float())
        R.matmul_wgrad(ref, A, B, accumulate=True)
    A, B = A.to(DEV), B.to(DEV)
    lda, ldb = A.stride(0) if A.shape[0] > 1 else A.shape[1], B.stride(0) if B.shape[0] > 1 else B.shape[1]
    rc = _lib.cuda().llmc_gemm_tiled(KN._p(A), KN._p(B), KN._p(out), KN._p(bias), KN._p(pre), M, N, K, lda, ldb, N, a_mn, b_mn, md, 1, 1,
                                     ctypes.c_void_p(0), ctypes.c_void_p(0), 0, bn, KN._stream())
    assert rc == 0
    close(out[:M], ref, 3e-2, 1.5e-2)              # sums of up to 776 products of size 0.05, rounded to bf16 once or twice
    if mode == "gelu":
        close(pre, refpre, 2e-2, 1e-2)
    assert (out[M:] == 7.0).all() and _lib.read_status() == 0
