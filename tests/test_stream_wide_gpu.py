"""Streaming products with several weight tiles per CTA (the LM head of a decoding step): one more tile than CTAs, ragged columns and depths, every
accumulator width, and their form with fp32 logits and a counter."""
import ctypes

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


# a CTA per tile and several tiles per CTA; columns that end with the rows of the weights, inside a tile on any remainder of 4, and tiles before their end
@pytest.mark.parametrize("M", [1, 17, 128])
@pytest.mark.parametrize("N,cols,K", [(512, 500, 64), (512, 301, 1024), (296 * 128 + 200, 296 * 128 + 131, 72), (50304, 50257, 768), (3 * 296 * 128, 2 * 296 * 128 + 2, 64)])
def test_logits_and_counter(M, N, cols, K):
    lib = _lib.cuda()
    entry = lib.llmc_stream_gemm_logits
    entry.restype, entry.argtypes = ctypes.c_int, [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p] + [ctypes.c_int] * 5 + [ctypes.c_void_p] * 2
    g = torch.Generator(device=DEV).manual_seed(M + N)
    x, w = torch.randn(M, K, generator=g, device=DEV).bfloat16(), (torch.randn(N, K, generator=g, device=DEV) * 0.1).bfloat16()
    want = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    assert lib.llmc_stream_gemm(KN._p(want), KN._p(x), KN._p(w), KN._p(None), M, N, K, K, K, N, 0, KN._stream()) == 0
    out, at = torch.full((M * cols + 300,), 7.0, device=DEV), torch.tensor([41, 5], dtype=torch.int32, device=DEV)
    for counter in (at, None):
        out[:M * cols] = -1.0
        assert entry(KN._p(out), cols, KN._p(x), KN._p(w), M, N, K, K, K, KN._p(counter), KN._stream()) == 0
        # the bits of the bf16 form, rows of `cols`, nothing behind them
        assert torch.equal(out[:M * cols].view(M, cols), want[:, :cols].float()) and (out[M * cols:] == 7.0).all()
        assert at.tolist() == [42, 5]
    assert _lib.read_status() == 0
