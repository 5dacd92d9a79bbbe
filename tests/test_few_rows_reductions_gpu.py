"""Bias gradients of few rows (one launch, no scratch), around the line to the two-launch form; the two parts of the LayerNorm backward."""
import contextlib

import pytest
import torch

from llmc_b200.ops import kernels as KN

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows", [1, 63, 65, 256, 1000, 1024, 1025])
@pytest.mark.parametrize("OC", [8, 40, 2304])
@pytest.mark.parametrize("accumulate", [False, True])
def test_bias_grad(rows, OC, accumulate):
    g = torch.Generator(device=DEV).manual_seed(rows + OC)
    d, old = torch.randn(rows, OC, generator=g, device=DEV).bfloat16(), torch.randn(OC, generator=g, device=DEV).bfloat16()
    buf = torch.full((OC + 8,), 7.0, dtype=torch.bfloat16, device=DEV)
    buf[:OC] = old
    KN.bias_grad(buf[:OC], d, accumulate=accumulate)
    want = d.double().sum(0) + (old.double() if accumulate else 0.0)
    # one rounding to bf16; fp32 sums of up to 1025 terms of size 1
    assert not ((buf[:OC].double() - want).abs() > 1e-3 + want.abs() * 2 ** -8).any()
    assert (buf[OC:] == 7.0).all()


@pytest.mark.parametrize("rows,OC", [(3, 65536), (3, 65544), (834, 50304), (833, 50304)])
def test_bias_grad_of_wide_outputs(rows, OC):
    g = torch.Generator(device=DEV).manual_seed(rows + OC)
    d, out = torch.randn(rows, OC, generator=g, device=DEV).bfloat16(), torch.full((OC + 8,), 7.0, dtype=torch.bfloat16, device=DEV)
    KN.bias_grad(out[:OC], d, accumulate=False)
    want = d.double().sum(0)
    assert not ((out[:OC].double() - want).abs() > 1e-3 + want.abs() * 2 ** -8).any() and (out[OC:] == 7.0).all()


def test_layernorm_backward_in_two_streams():
    N, C = 300, 384
    g = torch.Generator(device=DEV).manual_seed(1)
    n = lambda *s: torch.randn(*s, generator=g, device=DEV).bfloat16()
    dout, inp, w, b = n(N, C), n(N, C), n(C), n(C)
    out, mean, rstd = torch.empty_like(inp), torch.empty(N, device=DEV), torch.empty(N, device=DEV)
    KN.layernorm_forward(out, mean, rstd, inp, w, b)
    res = []
    for other in (False, True):
        dinp, dw, db, dc = torch.ones_like(inp), torch.ones_like(w), torch.ones_like(w), torch.ones_like(w)
        side = torch.cuda.Stream()

        @contextlib.contextmanager
        def elsewhere():
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                yield
        KN.layernorm_backward(dinp, dw, db, dout, inp, w, mean, rstd, dcolsum=dc, sums_in=elsewhere if other else None)
        torch.cuda.synchronize()
        res.append((dinp, dw, db, dc))
    assert all(torch.equal(x, y) for x, y in zip(*res))
