"""Generation with a key / value cache on the CPU path: cached logits against the training forward pass, batched prompts of
different lengths, stop tokens, echo, nucleus sampling (behaviour of LLaMA.generate / sample_top_p in the reference's
train_llama3.py:476-576)."""
import pytest
import torch

from llmc_b200.models import generate as G
from llmc_b200.models import llama3
from llmc_b200.ops import kernels as KN

DESC = "llama3:l=2,c=64,h=4,kv=2,t=48,v=97,m=32,f=1.0"


def small_model(desc=DESC):
    m = llama3.Llama(llama3.config_from_descriptor(desc), "cpu", torch.float32, recompute=0)
    m.init_random(7)
    for n in ("qkvw", "attprojw", "fc12w", "fcprojw", "lmhead"):
        m.params[n].mul_(4.0)
    return m


def test_cached_logits_match_full_forward():
    m = small_model()
    g = torch.Generator().manual_seed(0)
    B, T = 3, 20
    tok = torch.randint(0, m.cfg.vocab_size, (B, T), generator=g, dtype=torch.int32)
    m.forward(tok)
    full = m.logits()[..., :m.cfg.vocab_size].clone()                 # (B, T, V)
    dec = G.CachedDecoder(m, B, 32)
    got = dec.forward(tok[:, :7].contiguous(), 0)                     # prefill of 7 tokens
    assert torch.allclose(got, full[:, 6], atol=1e-4, rtol=1e-4)
    got = dec.forward(tok[:, 7:10].contiguous(), 7)                   # three at once
    assert torch.allclose(got, full[:, 9], atol=1e-4, rtol=1e-4)
    for t in range(10, T):                                            # then one by one
        got = dec.forward(tok[:, t:t + 1].contiguous(), t)
        assert torch.allclose(got, full[:, t], atol=1e-4, rtol=1e-4), "position %d" % t


def test_dense_prefill_fills_the_cache_like_the_incremental_path():
    m = small_model()
    g = torch.Generator().manual_seed(1)
    tok = torch.randint(0, m.cfg.vocab_size, (2, 24), generator=g, dtype=torch.int32)
    a, b = G.CachedDecoder(m, 2, 32), G.CachedDecoder(m, 2, 32)
    a.dense_prefill_from, b.dense_prefill_from = 8, 1000
    la, lb = a.forward(tok[:, :20].contiguous(), 0), b.forward(tok[:, :20].contiguous(), 0)
    assert torch.allclose(la, lb, atol=1e-5, rtol=1e-5)
    assert torch.allclose(a.kcache, b.kcache, atol=1e-6) and torch.allclose(a.vcache, b.vcache, atol=1e-6)
    for t in range(20, 24):
        la, lb = a.forward(tok[:, t:t + 1].contiguous(), t), b.forward(tok[:, t:t + 1].contiguous(), t)
    assert torch.allclose(la, lb, atol=1e-5, rtol=1e-5)


def test_single_kv_head_and_full_heads():
    for desc in ("llama3:l=1,c=64,h=4,kv=1,t=32,v=50,m=16,f=1.0", "llama3:l=1,c=64,h=4,kv=4,t=32,v=50,m=16,f=1.3"):
        m = small_model(desc)
        tok = torch.arange(24, dtype=torch.int32).view(2, 12) % m.cfg.vocab_size
        m.forward(tok)
        full = m.logits()[..., :m.cfg.vocab_size].clone()
        dec = G.CachedDecoder(m, 2, 16)
        dec.forward(tok[:, :5].contiguous(), 0)
        for t in range(5, 12):
            got = dec.forward(tok[:, t:t + 1].contiguous(), t)
        assert torch.allclose(got, full[:, 11], atol=1e-4, rtol=1e-4)


def test_generate_cache_equals_recompute_and_forces_prompts():
    m = small_model()
    prompts = [[5, 9, 11, 3], [7, 2], [1, 2, 3, 4, 5, 6, 8]]
    with_cache = G.generate(m, prompts, max_gen_len=10, temperature=0.0, echo=True)
    without = G.generate(m, prompts, max_gen_len=10, temperature=0.0, echo=True, use_kv=False)
    assert with_cache == without
    for p, out in zip(prompts, with_cache):
        assert out[:len(p)] == p
        assert len(out) <= len(p) + 10
    # every row continues as it would alone: batching must not leak between rows
    for p, out in zip(prompts, with_cache):
        alone = G.generate(m, [p], max_gen_len=10, temperature=0.0, echo=True)[0]
        n = min(len(alone), len(out))
        assert alone[:n] == out[:n]
    no_echo = G.generate(m, prompts, max_gen_len=10, temperature=0.0)
    for p, full, tail in zip(prompts, with_cache, no_echo):
        assert full[len(p):] == tail


def test_stop_tokens_cut_the_output_and_end_the_loop():
    m = small_model()
    prompts = [[5, 9, 11, 3], [7, 2]]
    free = G.generate(m, prompts, max_gen_len=12, temperature=0.0)
    stop = free[0][2]                                                  # a token the first row is known to produce
    cut = G.generate(m, prompts, max_gen_len=12, temperature=0.0, stop_tokens=(stop,))
    assert cut[0] == free[0][:free[0].index(stop)]
    assert stop not in cut[1]
    assert free[1][:len(cut[1])] == cut[1]


def test_context_window_bounds_generation():
    m = small_model()
    out = G.generate(m, [list(range(1, 41))], max_gen_len=100, temperature=0.0, echo=True)[0]
    assert len(out) == m.cfg.max_seq_len


def test_sample_top_p():
    g = torch.Generator().manual_seed(0)
    probs = torch.tensor([[0.5, 0.3, 0.15, 0.05]]).repeat(4000, 1)
    picks = G.sample_top_p(probs, 0.7, g)                              # nucleus = {0, 1}: mass before token 2 is 0.8 > 0.7
    counts = torch.bincount(picks, minlength=4).float() / 4000
    assert counts[2] == 0 and counts[3] == 0
    assert abs(counts[0] - 0.625) < 0.03 and abs(counts[1] - 0.375) < 0.03
    assert torch.equal(G.sample_top_p(probs[:8], 0.0, g), torch.zeros(8, dtype=torch.int64))   # only the top token survives
    g1, g2 = torch.Generator().manual_seed(3), torch.Generator().manual_seed(3)
    m = small_model()
    a = G.generate(m, [[4, 5, 6]], 8, temperature=0.8, top_p=0.9, generator=g1)
    b = G.generate(m, [[4, 5, 6]], 8, temperature=0.8, top_p=0.9, generator=g2)
    assert a == b


def test_products_stay_inside_their_outputs(monkeypatch):
    """Whole-tile products of a batch of more than one tile: as many rows of the output as of the input, whatever was run before."""
    m = small_model("llama3:l=1,c=64,h=4,kv=2,t=64,v=97,m=32,f=1.0")
    shapes = []
    product = G.ops.matmul_forward

    def spy(out, inp, weight, bias):
        shapes.append((out.shape[0], inp.shape[0]))
        product(out, inp, weight, bias)

    monkeypatch.setattr(G.ops, "matmul_forward", spy)
    g = torch.Generator().manual_seed(0)
    dec, plain = G.CachedDecoder(m, 200, 16), G.CachedDecoder(m, 200, 16)
    dec.whole_tiles = True
    # a batch of several tiles after a longer prompt, and a batch that grows from call to call
    for B, T in ((129, 10), (129, 1), (3, 2), (200, 1), (200, 3), (130, 1)):
        tok = torch.randint(0, m.cfg.vocab_size, (B, T), generator=g, dtype=torch.int32)
        shapes.clear()
        got = dec.forward(tok, 0)
        rows, last = (B * T + 127) // 128 * 128, (B + 127) // 128 * 128
        assert shapes == [(rows, rows)] * 4 + [(last, last)]
        assert torch.allclose(got, plain.forward(tok, 0), atol=1e-4, rtol=1e-4)


@pytest.mark.parametrize("op,shapes", [
    ("matmul_forward", [(255, 64), (256, 32), (64, 32)]), ("matmul_forward", [(256, 56), (256, 32), (64, 32)]),
    ("matmul_forward", [(256, 64), (256, 32), (64, 24)]), ("matmul_forward", [(256, 64), (256, 32), (64, 32), (56,)]),
    ("matmul_forward", [(256, 64), (256, 32), (64, 32), (64,), (255, 64)]),
    ("matmul_dgrad", [(255, 32), (256, 64), (64, 32)]), ("matmul_dgrad", [(256, 32), (256, 64), (56, 32)]),
    ("matmul_dgrad", [(256, 32), (256, 64), (64, 32), (255, 32)]),
    ("matmul_wgrad", [(56, 32), (256, 64), (256, 32)]), ("matmul_wgrad", [(64, 32), (256, 64), (255, 32)]),
    ("matmul_skinny", [(7, 64), (8, 32), (64, 32)]), ("matmul_skinny", [(8, 56), (8, 32), (64, 32)]), ("matmul_skinny", [(8, 64), (8, 32), (64, 24)]),
    ("matmul_swiglu", [(7, 64), (8, 32), (128, 32)]), ("matmul_swiglu", [(8, 56), (8, 32), (128, 32)]), ("matmul_swiglu", [(8, 64), (8, 32), (128, 24)])])
def test_device_products_refuse_operands_that_are_too_small(monkeypatch, op, shapes):
    """The launchers raise before anything is launched."""
    def library():
        raise AssertionError("launched")
    monkeypatch.setattr(KN._lib, "cuda", library)
    with pytest.raises(ValueError):
        getattr(KN, op)(*[torch.zeros(*s, dtype=torch.bfloat16) for s in shapes])


@pytest.mark.parametrize("M,N,K", [(0, 64, 64), (4, 0, 64), (4, 64, 0)])
def test_an_empty_product_of_few_rows_is_no_error(M, N, K):
    """All three product kernels return without a launch (no GPU is needed for that)."""
    lib = KN._lib.cuda()
    assert lib.llmc_stream_gemm(None, None, None, None, M, N, K, 64, 64, 64, 0, None) == 0
    assert lib.llmc_gemm(None, None, None, None, None, M, N, K, 64, 64, 64, 0, 0, KN.MODE_STORE, 0, 1, None, None, 0, None) == 0
    assert lib.llmc_gemm2(None, None, None, None, None, M, N, K, 64, 64, 64, 0, 0, KN.MODE_STORE, 0, 1, None, None, None) == 0


def spread(t, dim):
    """The same values with a gap behind every slice of ``dim``."""
    shape = list(t.shape)
    shape[dim] += 3
    big = torch.zeros(shape, dtype=t.dtype)
    out = big.narrow(dim, 0, t.shape[dim])
    out.copy_(t)
    assert not out.is_contiguous()
    return out


@pytest.mark.parametrize("what", ["plain", "kcache", "vcache", "qkvw", "fcprojw", "short lmhead"])
def test_the_natively_issued_pass_gets_only_layers_at_equal_distances(monkeypatch, what):
    m = small_model()
    tok = torch.arange(14, dtype=torch.int32).view(2, 7)
    want = G.CachedDecoder(m, 2, 32).forward(tok, 0)
    dec, issued = G.CachedDecoder(m, 2, 32), []
    dec.native, dec.skinny_rows = True, KN.STREAM_MAX_ROWS     # as for a bf16 model on the GPU
    monkeypatch.setattr(KN, "decoder_forward", lambda *a: issued.append(a))
    if what.endswith("cache"):
        setattr(dec, what, spread(getattr(dec, what), 1))
    elif what == "short lmhead":                               # fewer rows than the buffer of logits has columns
        m.params["lmhead"] = m.params["lmhead"][:-8]
    elif what != "plain":
        m.params[what] = spread(m.params[what], m.params[what].dim() - 2)
    if what == "short lmhead":
        with pytest.raises((RuntimeError, ValueError)):
            dec.forward(tok, 0)
    else:
        got = dec.forward(tok, 0)
        assert what == "plain" or torch.allclose(got, want, atol=1e-5, rtol=1e-5)
    assert len(issued) == (what == "plain")
