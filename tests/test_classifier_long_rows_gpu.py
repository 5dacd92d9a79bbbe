"""Softmax, loss and gradient of logits on both sides of the row length from which on a row has more threads."""
import pytest
import torch

from llmc_b200 import _lib
from llmc_b200.ops import kernels as KN

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("N,V,Vp", [(3, 61440, 61440), (3, 61441, 61448), (2, 61448, 61448), (300, 70001, 70016), (5, 128256, 128256), (1, 200003, 200064)])
def test_against_64_bits(N, V, Vp):
    g = torch.Generator(device=DEV).manual_seed(Vp + N)
    x = (torch.randn(N, Vp, generator=g, device=DEV) * 3).bfloat16()
    x[0, 0], x[0, V - 1], x[-1, V // 2] = 40.0, -float("inf"), 30.0
    x[:, V:] = float("nan")                                     # padding is not read
    t = torch.randint(0, V, (N,), generator=g, device=DEV, dtype=torch.int32)
    t[-1] = V - 1 if N > 1 else 0
    d, losses, again, lossa = x.clone(), torch.zeros(N, device=DEV), x.clone(), torch.ones(N, device=DEV)
    KN.fused_classifier(d, losses, t, 0.5, V, True, False)
    KN.fused_classifier(again, lossa, t, 0.5, V, False, True)
    assert _lib.read_status() == 0
    ref = torch.log_softmax(x[:, :V].double(), -1)
    loss = -ref.gather(1, t.long()[:, None])[:, 0]
    # exponentials good to 2^-22, their sum in 32 bits: far below 1e-4 of a loss of about 15
    assert torch.allclose(losses.double(), loss, atol=1e-4) and torch.allclose(lossa.double(), loss + 1, atol=1e-4)
    assert torch.equal(torch.nan_to_num(again, 7.0), torch.nan_to_num(x, 7.0))
    p = ref.exp()
    p[torch.arange(N), t.long()] -= 1
    # the gradient is rounded to bf16 once: half a unit in the last of 8 places, 2^-8 of each element; before that exponents up to 60 are rounded to 32 bits, 2^-18 of
    # the result twice (here and in the maximum), and the target's difference has an absolute error of 2^-24
    assert ((d[:, :V].double() - 0.5 * p).abs() <= (2 ** -8 + 2 ** -16) * (0.5 * p).abs() + 2 ** -24 * (p < 0)).all()
    assert (d[:, V:] == 0).all()
