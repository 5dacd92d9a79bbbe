"""The natively issued decoder pass against the same operators called one by one: prompts below and above the dense and the 128-row line, one-token
steps, chunks in the middle of the cache."""
import pytest
import torch

from llmc_b200.models import generate, llama3
from llmc_b200.ops import kernels as KN

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


# hidden widths 1024 (either fused MLP), 224 (neither) and 576 (the streamed one only), channels from which the swapped products start
@pytest.mark.parametrize("desc", ["llama3:l=2,c=256,h=4,kv=2,t=2048,v=500", "llama3:l=2,c=256,h=4,kv=4,t=2048,v=500,m=32,f=0.3",
                                  "llama3:l=1,c=256,h=2,kv=1,t=2048,v=500,m=32,f=0.8", "llama3:l=2,c=768,h=12,kv=4,t=2048,v=500"])
@pytest.mark.parametrize("B,chunks", [(1, [7, 1, 1]), (3, [40, 1, 5]), (2, [70, 3]), (1, [128, 1]), (2, [200, 130]), (130, [2, 1]), (3, [777, 1])])
def test_same_logits_and_cache(desc, B, chunks):
    m = llama3.Llama(llama3.config_from_descriptor(desc), DEV, torch.bfloat16)
    m.init_random(3)
    # 20 instead of 800 positions for 130 rows: neither is more than a few hundred MB
    fast, slow = (generate.CachedDecoder(m, B, 800 if B < 100 else 20) for _ in range(2))
    slow.native, slow.whole_tiles = False, False               # the operators one by one, on exactly the same rows
    g = torch.Generator().manual_seed(1)
    at = 0
    for n in chunks:
        tok = torch.randint(0, 500, (B, n), generator=g, dtype=torch.int32).to(DEV)
        before = KN.launch_count()
        a = fast.forward(tok, at)
        issued = KN.launch_count() - before
        b = slow.forward(tok, at)
        assert issued == KN.launch_count() - before - issued
        at += n
        # the same kernels on the same rows: the same bits
        assert torch.equal(a, b) and torch.equal(fast.kcache, slow.kcache) and torch.equal(fast.vcache, slow.vcache)
        assert torch.isfinite(a).all() and a.abs().max() > 0


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
    assert torch.equal(got, want) and torch.equal(apart.kcache, plain.kcache) and torch.equal(apart.vcache, plain.vcache)
    assert not around[:, 2:].any()


# a head of one weight tile per CTA, and of several
@pytest.mark.parametrize("vocab", [500, 50001])
def test_replayed_steps(vocab):
    m = llama3.Llama(llama3.config_from_descriptor("llama3:l=2,c=256,h=4,kv=2,t=256,v=%d" % vocab), DEV, torch.bfloat16)
    m.init_random(3)
    replayed, launched = generate.CachedDecoder(m, 3, 64), generate.CachedDecoder(m, 3, 64)
    tok = torch.randint(0, vocab, (3, 20), generator=torch.Generator().manual_seed(1), dtype=torch.int32).to(DEV)
    for d in (replayed, launched):
        d.forward(tok[:, :15].contiguous(), 0)
    step = generate.GraphStep(replayed, 3, 15)
    for i in range(15, 20):
        got, want = step.step(tok[:, i:i + 1].contiguous()), launched.forward(tok[:, i:i + 1].contiguous(), i)
        assert torch.equal(got, want) and got.shape == (3, vocab) and int(step.pos) == i + 1
    assert torch.equal(replayed.kcache[:, :, :20], launched.kcache[:, :, :20]) and torch.equal(replayed.vcache[:, :, :20], launched.vcache[:, :, :20])
