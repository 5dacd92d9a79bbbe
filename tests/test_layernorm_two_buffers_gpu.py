"""LayerNorm backward that adds to one buffer and writes another gives the bits of the one in place, and leaves its input alone."""
import pytest
import torch

from llmc_b200 import _lib, ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("N,C", [(1, 8), (300, 768), (257, 4096)])
def test_two_buffers(N, C, dtype):
    g = torch.Generator().manual_seed(N + C)
    old, dout, inp = [torch.randn(N, C, generator=g).to(dtype).to(DEV) for _ in range(3)]
    w = torch.randn(C, generator=g).to(dtype).to(DEV)
    mean, rstd = inp.float().mean(1), (inp.float().var(1, unbiased=False) + 1e-5).rsqrt()
    new = lambda: torch.zeros(C, dtype=dtype, device=DEV)
    a, b = [new(), new(), new()], [new(), new(), new()]
    inplace, out, kept = old.clone(), torch.full((N + 1, C), 7.0, dtype=dtype, device=DEV), old.clone()
    ops.layernorm_backward(inplace, a[0], a[1], dout, inp, w, mean, rstd, dcolsum=a[2])
    ops.layernorm_backward(out[:N], b[0], b[1], dout, inp, w, mean, rstd, dcolsum=b[2], dinp_old=old)
    assert torch.equal(out[:N], inplace) and torch.equal(old, kept) and (out[N:] == 7.0).all() and _lib.read_status() == 0
    assert all(torch.equal(x, y) for x, y in zip(a, b))
