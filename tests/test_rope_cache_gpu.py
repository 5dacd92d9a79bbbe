"""The rotary kernel's second destination: rotated keys and values enter the cache as they enter the packed tensor, nothing else of the cache changes."""
import pytest
import torch

from llmc_b200.ops import kernels as KN
from llmc_b200.ops import reference as R

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("NH,NKV", [(4, 4), (4, 2), (6, 2), (8, 2)])
@pytest.mark.parametrize("B,T,cache_len,HS", [(1, 5, 5, 64), (3, 37, 50, 128)])
def test_cache_entries(B, T, cache_len, HS, NH, NKV):
    g = torch.Generator().manual_seed(NH * T + NKV)
    raw, freqs = torch.randn(B * T, (NH + 2 * NKV) * HS, generator=g).bfloat16(), torch.randn(T, HS // 2, 2, generator=g)
    packed = torch.empty(B * T, 3 * NH * HS, dtype=torch.bfloat16, device=DEV)
    kc, vc = (torch.full((B + 1, cache_len, NKV, HS), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    KN.rope_forward(packed, raw.to(DEV), freqs.to(DEV), T, NH, NKV, kc, vc)
    x = packed.view(B, T, 3, NKV, NH // NKV, HS)
    plain = torch.empty_like(packed)
    KN.rope_forward(plain, raw.to(DEV), freqs.to(DEV), T, NH, NKV)
    assert torch.equal(packed, plain)
    for c, which in ((kc, 1), (vc, 2)):
        assert torch.equal(c[:B, :T], x[:, :, which, :, 0])
        assert (c[B:] == 7.0).all() and (c[:, T:] == 7.0).all()
    rp, rk, rv = torch.empty(B * T, 3 * NH * HS), torch.empty(B, cache_len, NKV, HS), torch.empty(B, cache_len, NKV, HS)
    R.rope_forward(rp, raw, freqs, T, NH, NKV, rk, rv)
    # a product sum of two terms, rounded once
    assert not ((kc[:B, :T].cpu().float() - rk[:, :T]).abs() > 2e-2 + 2 ** -7 * rk[:, :T].abs()).any()
    assert torch.equal(vc[:B, :T].cpu().float(), rv[:, :T])


def test_refuses_a_cache_that_is_too_small():
    z = lambda *s: torch.zeros(*s, dtype=torch.bfloat16, device=DEV)
    for kc in (z(1, 4, 2, 64), z(2, 3, 2, 64), z(2, 4, 1, 64)):
        with pytest.raises(ValueError):
            KN.rope_forward(z(8, 3 * 4 * 64), z(8, 8 * 64), torch.zeros(4, 32, 2, device=DEV), 4, 4, 2, kc, kc.clone())
