"""Streaming products with several weight tiles per CTA (the LM head of a decoding step): one more tile than CTAs, ragged columns and depths, every
accumulator width."""
import pytest
import torch

from llmc_b200 import _lib
from llmc_b200.ops import kernels as KN

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("M", [1, 16, 17, 40, 100, 128])
@pytest.mark.parametrize("N,K,bias", [(296 * 128 + 8, 72, True), (50304, 768, False), (3 * 296 * 128, 64, False)])
def test_wide_output(M, N, K, bias):
    if 2 * KN.sm_count(torch.device(DEV, 0)) * 128 >= N:
        pytest.skip("a CTA per tile on this device")
    g = torch.Generator(device=DEV).manual_seed(M + N)
    x, w = torch.randn(M, K, generator=g, device=DEV).bfloat16(), (torch.randn(N, K, generator=g, device=DEV) * 0.1).bfloat16()
    b = torch.randn(N, generator=g, device=DEV).bfloat16() if bias else None
    out = torch.full((M + 2, N), 7.0, dtype=torch.bfloat16, device=DEV)
    assert _lib.cuda().llmc_stream_gemm(KN._p(out), KN._p(x), KN._p(w), KN._p(b), M, N, K, K, K, N, 0, KN._stream()) == 0
    want = x.double() @ w.double().t() + (b.double() if bias else 0.0)
    # one rounding to bf16 of a sum that is exact to fp32
    assert not ((out[:M].double() - want).abs() > 1e-3 + want.abs() * 2 ** -8).any()
    assert (out[M:] == 7.0).all() and _lib.read_status() == 0
