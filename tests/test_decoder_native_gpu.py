"""The natively issued decoder pass against the same operators called one by one: prompts below and above the dense and the 128-row line, one-token
steps, chunks in the middle of the cache."""
import pytest
import torch

from llmc_b200.models import generate, llama3
from llmc_b200.ops import kernels as KN

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


# hidden widths 1024 (either fused MLP), 224 (neither) and 576 (the streamed one only)
@pytest.mark.parametrize("desc", ["llama3:l=2,c=256,h=4,kv=2,t=512,v=500", "llama3:l=2,c=256,h=4,kv=4,t=512,v=500,m=32,f=0.3", "llama3:l=1,c=256,h=2,kv=1,t=512,v=500,m=32,f=0.8"])
@pytest.mark.parametrize("B,chunks", [(1, [7, 1, 1]), (3, [40, 1, 5]), (2, [70, 3]), (1, [128, 1]), (2, [200, 130]), (130, [2, 1])])
def test_same_logits_and_cache(desc, B, chunks):
    m = llama3.Llama(llama3.config_from_descriptor(desc), DEV, torch.bfloat16)
    m.init_random(3)
    fast, slow = generate.CachedDecoder(m, B, 400), generate.CachedDecoder(m, B, 400)
    called = []
    slow.skinny_rows = 127                                    # not the default: the operators one by one
    g = torch.Generator().manual_seed(1)
    at = 0
    for n in chunks:
        tok = torch.randint(0, 500, (B, n), generator=g, dtype=torch.int32).to(DEV)
        before = KN.launch_count()
        a = fast.forward(tok, at)
        called.append(KN.launch_count() - before)
        b = slow.forward(tok, at)
        at += n
        for x, y in ((a, b), (fast.kcache, slow.kcache), (fast.vcache, slow.vcache)):
            # the same kernels but for products of exactly 128 rows and row tiles: bf16 roundings of two layers apart
            assert float((x.float() - y.float()).norm() / y.float().norm()) < 1e-2
    assert min(called) > 0


def test_layers_that_lie_apart():
    """Caches and weights with a gap behind every layer are read one layer at a time."""
    m = llama3.Llama(llama3.config_from_descriptor("llama3:l=2,c=256,h=4,kv=2,t=512,v=500"), DEV, torch.bfloat16)
    m.init_random(3)
    tok = torch.randint(0, 500, (2, 9), generator=torch.Generator().manual_seed(1), dtype=torch.int32).to(DEV)
    plain, apart = generate.CachedDecoder(m, 2, 64), generate.CachedDecoder(m, 2, 64)
    want = plain.forward(tok, 0)
    around = torch.zeros(2, 4, *apart.kcache.shape[2:], dtype=torch.bfloat16, device=DEV)
    apart.kcache = around[:, :2]
    weights = torch.zeros(2, m.params["qkvw"].shape[1] + 8, 256, dtype=torch.bfloat16, device=DEV)
    weights[:, :-8] = m.params["qkvw"]
    m.params["qkvw"] = weights[:, :-8]
    got = apart.forward(tok, 0)
    for x, y in ((got, want), (apart.kcache, plain.kcache), (apart.vcache, plain.vcache)):
        assert float((x.float() - y.float()).norm() / y.float().norm()) < 1e-2
    assert not around[:, 2:].any()
