"""Replayed micro-steps give the bits of launched ones: over gradient accumulation, a change of shape, and scratch buffers that other
callers outgrow in between."""
import pytest
import torch

from llmc_b200.models import gpt2, llama3
from llmc_b200.ops import kernels as KN
from llmc_b200.parallel.dist import DistConfig
from llmc_b200.parallel.zero import ShardedAdamW

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def make(family):
    if family == "gpt2":
        return gpt2.GPT(gpt2.GPTConfig(64, 1000, 1024, 2, 2, 128), DEV, torch.bfloat16, recompute=1)
    return llama3.Llama(llama3.config_from_descriptor("llama3:l=2,c=256,h=4,kv=2,t=64,v=500,m=64,f=1.0"), DEV, torch.bfloat16)


def train(family, use_graphs):
    m = make(family)
    m.init_random(3)
    m.use_graphs = use_graphs
    opt = ShardedAdamW(m, DistConfig(0, 1, 0, DEV), 0, True)
    g = torch.Generator().manual_seed(0)
    seen, counts = [], []
    for step in range(10):
        T = 40 if step == 6 else 64
        before = KN.launch_count()
        for micro in range(2):
            tok = torch.randint(0, 500, (2, T + 1), generator=g, dtype=torch.int32)
            m.forward(tok[:, :-1].contiguous().to(DEV), tok[:, 1:].contiguous().to(DEV), 2, micro)
            m.backward(micro, micro == 1)
        counts.append(KN.launch_count() - before)
        seen += [m.loss(2).clone(), m.grads_flat.clone()]
        if step == 4:                                          # another caller needs larger scratch buffers
            big = torch.zeros(4096, 4096, dtype=torch.bfloat16, device=DEV)
            KN.bias_grad(torch.zeros(4096, dtype=torch.bfloat16, device=DEV), big)
            KN.matmul_wgrad(torch.zeros(512, 512, dtype=torch.bfloat16, device=DEV), big[:, :512].contiguous(), big[:, 512:1024].contiguous())
        opt.grad_norm_sq()
        opt.step(3e-3, 0.1, step + 1)
    return seen + [m.params_flat.clone()], counts, m


@pytest.mark.parametrize("family", ["gpt2", "llama3"])
def test_replayed_steps_equal_launched_steps(family):
    other = KN._scratch.get("another_caller", 1000, torch.float32, DEV)
    want, launches, _ = train(family, False)
    got, counted, m = train(family, True)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert counted == launches
    graphs = [e for e in m.step_graphs._entries.values() if e["graph"] is not None]
    assert graphs
    assert all(len(e["scratch"]) > 0 and not any(t is other for t in e["scratch"]) for k, e in m.step_graphs._entries.items() if k[0] == "backward" and e["graph"])


# 256 rows of 768 channels: input gradients in slices of K beside the weight gradients; 1280 rows: bias gradients through a scratch buffer, on the side
# branch; 2048 rows: the chain without priority over the side branches; every recompute level shares other buffers between the layers
@pytest.mark.parametrize("recompute", [0, 1, 2])
@pytest.mark.parametrize("B,T,C,L", [(4, 64, 768, 3), (5, 256, 256, 4), (8, 256, 256, 3)])
@pytest.mark.parametrize("family", ["gpt2", "llama3"])
def test_both_branches_of_the_backward_pass(family, B, T, C, L, recompute):
    def build(graphs):
        if family == "gpt2":
            m = gpt2.GPT(gpt2.GPTConfig(T, 1000, 1024, L, C // 64, C), DEV, torch.bfloat16, recompute=recompute)
        else:
            m = llama3.Llama(llama3.config_from_descriptor("llama3:l=%d,c=%d,h=%d,kv=%d,t=%d,v=1000,m=64,f=1.0" % (L, C, C // 64, C // 128, T)), DEV, torch.bfloat16,
                             recompute=recompute)
        m.init_random(3)
        m.use_graphs = graphs
        return m

    replayed, launched = build(True), build(False)
    g = torch.Generator().manual_seed(0)
    for step in range(8):
        for micro in range(2):
            tok = torch.randint(0, 1000, (B, T + 1), generator=g, dtype=torch.int32)
            x, y = tok[:, :-1].contiguous().to(DEV), tok[:, 1:].contiguous().to(DEV)
            for m in (replayed, launched):
                m.forward(x, y, 2, micro)
                m.backward(micro, micro == 1)
            assert torch.equal(replayed.grads_flat, launched.grads_flat), (step, micro)
            assert torch.equal(replayed.acts["dresidual"], launched.acts["dresidual"])
        assert torch.equal(replayed.loss(2), launched.loss(2)) and torch.isfinite(launched.loss(2))
    assert sum(e["graph"] is not None for e in replayed.step_graphs._entries.values()) == 4
