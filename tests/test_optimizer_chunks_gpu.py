"""Gradient norm and AdamW over lists of chunks: slices shorter than, as long as and longer than a chunk, views of one element group, many layers, more chunks than
blocks."""
import pytest
import torch

from llmc_b200 import _lib
from llmc_b200.ops import kernels as KN

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _views(sizes, shift):
    """sizes: (elements of a slice, layers); shift: of every view in the optimizer's buffers (odd: the element-wise kernel)."""
    views, p, o = [], 0, shift
    for i, (n, L) in enumerate(sizes):
        views.append(dict(p_base=p, p_stride=n + 8, o_base=o, o_stride=n, n=n, L=L, wd=0.1 * (i % 2), seed=77 + i))
        p += (n + 8) * L
        o += n * L
    return views, p, o


@pytest.mark.parametrize("sizes", [
    [(8, 1)], [(1016, 3), (1024, 2), (1032, 2)], [(8, 40), (8192, 3), (8200, 2), (768, 12)], [(3 * 1024 * 1024 + 8, 2), (16, 1)],
    [(8 * (i + 1), 1 + i % 3) for i in range(16)],
    # 16 blocks of an SM share the norm's chunks of 8192 elements, 512 the update's of 1024: on 148 SMs a block takes a second one beyond 19.4 and 77.6
    # million elements, here in another view with slices of another length
    [(1000 * 1024 + 8, 30), (768, 40), (8200, 3), (8 * 1024 * 1024 + 16, 7), (1016, 5)]])
@pytest.mark.parametrize("master", [True, False])
def test_chunks(sizes, master):
    g = torch.Generator(device=DEV).manual_seed(len(sizes))
    views, P, O = _views(sizes, 0)
    odd = _views(sizes, 1)[0]
    rand = lambda n: torch.randn(n, generator=g, device=DEV)
    params, grads = rand(P).bfloat16(), rand(P).bfloat16()
    m, v, w = rand(O), rand(O).square(), rand(O)
    cover = torch.zeros(P, dtype=torch.bool, device=DEV)
    for t in views:
        for l in range(t["L"]):
            cover[t["p_base"] + l * t["p_stride"]:][:t["n"]] = True
    norm = torch.empty(1, device=DEV)
    KN.global_norm_sq(norm, grads, views)
    want = grads.double()[cover].square().sum()
    assert abs(float(norm) / float(want) - 1) < 1e-5          # sums of 32-bit terms in a fixed tree
    got = []
    for vw, shift in ((views, 0), (odd, 1)):
        pad = lambda t: torch.cat([torch.full((shift,), 3.0, device=DEV), t])
        q, mm, vv, ww = params.clone(), pad(m), pad(v), pad(w)
        KN.adamw_update(q, ww if master else None, grads, mm, vv, vw, 1e-3, 0.9, 0.95, 1e-8, 3, 1.0, norm, 1.0)
        got.append((q, mm[shift:], vv[shift:], ww[shift:]))
    assert _lib.read_status() == 0
    # the chunked and the element-wise kernel evaluate the same expressions: the same bits, and nothing between the slices is touched
    assert all(torch.equal(a, b) for a, b in zip(*got))
    q = got[0][0]
    assert torch.equal(q[~cover], params[~cover]) and not torch.equal(q[cover], params[cover])
