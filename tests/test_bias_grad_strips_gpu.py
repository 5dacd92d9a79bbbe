"""Bias gradients in two launches: strips shorter than, as long as and longer than the rows that a warp has in flight, ragged numbers of columns and strips."""
import pytest
import torch

from llmc_b200 import _lib
from llmc_b200.ops import kernels as KN

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows,OC", [(1025, 8), (1025, 1152), (5000, 264), (65536, 24), (40000, 1600), (33333, 768), (30, 70000), (2000, 28680)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_sums(rows, OC, accumulate):
    assert _lib.cuda().llmc_bias_grad_scratch(rows, OC) > 0
    g = torch.Generator(device=DEV).manual_seed(rows + OC)
    d, db = torch.randn(rows, OC, generator=g, device=DEV).bfloat16(), torch.randn(OC + 8, generator=g, device=DEV).bfloat16()
    want = d.double().sum(0) + (db[:OC].double() if accumulate else 0)
    got = db.clone()
    KN.bias_grad(got[:OC], d, accumulate=accumulate)
    assert _lib.read_status() == 0 and torch.equal(got[OC:], db[OC:])
    # one rounding to bf16; sums of `rows` 32-bit terms of size 1 in a tree of a few hundred steps
    assert not ((got[:OC].double() - want).abs() > 2.0 ** -8 * want.abs() + 1e-6 * rows ** 0.5 * 30).any()
    again = db.clone()
    KN.bias_grad(again[:OC], d, accumulate=accumulate)
    assert torch.equal(again, got)
