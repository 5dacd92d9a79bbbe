"""Performance cases of the framework's GPU paths: training operators of GPT-2 / GPT-3 / LLaMA-3 blocks, a whole small training
micro-step, the optimizer update, and LLaMA-3 prefill and decoding.

``listed()`` gives the standing cases, ``draw(rng)`` one more of the same ranges; ``prepare`` / ``run`` execute one pass through the
public entry points (``llmc_b200.ops``, ``models``, ``parallel.zero``), ``exact`` restates the pass in float64 with plain torch.
Every input is drawn on the GPU from the case's seed."""
import math

import torch

DEV = "cuda"
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64


def listed():
    return [
        # causal attention of the GPT-2 124M benchmark micro-batch (64 x 1024 tokens, 12 heads of 64), forward and backward
        {"name": "attn_gpt2_124M", "kind": "attention", "B": 64, "T": 1024, "NH": 12, "HS": 64},
        # the GPT-3 2.7B head layout (32 heads of 80) on a ragged sequence length, small batch
        {"name": "attn_gpt3_ragged", "kind": "attention", "B": 3, "T": 1000, "NH": 32, "HS": 80},
        # rotary embedding + grouped-query attention of LLaMA-3 8B at 4096 tokens, forward and backward
        {"name": "gqa_llama_8B", "kind": "gqa", "B": 2, "T": 4096, "NH": 32, "NKV": 8, "HS": 128},
        # GPT-2 124M MLP (up-projection + GELU, down-projection) with both bias gradients, a later micro-step (gradients accumulate)
        {"name": "mlp_gpt2_124M", "kind": "mlp", "N": 65536, "C": 768, "accumulate": True},
        # LLaMA-3 8B SwiGLU MLP on an odd number of rows
        {"name": "mlp_llama_8B_ragged", "kind": "swiglu", "N": 3001, "C": 4096, "H": 14336, "accumulate": False},
        # residual add + LayerNorm between the sub-layers of GPT-2 124M and its backward with the projection's bias gradient
        {"name": "norm_gpt2_124M", "kind": "norm", "N": 65536, "C": 768, "rms": False},
        # LM head, fused softmax cross-entropy and both gradients of the tied embedding matrix
        {"name": "head_gpt2_124M", "kind": "head", "N": 16384, "C": 768, "V": 50257, "Vp": 50304},
        # gradient norm + AdamW with fp32 master weights over all tensors of GPT-2 124M
        {"name": "update_gpt2_124M", "kind": "update", "depth": 12},
        # whole forward + backward of GPT-2 124M on the 4 x 64 tokens of the reference's numerics test: launches and latency
        {"name": "step_gpt2_4x64", "kind": "step", "depth": 12, "B": 4, "T": 64, "dtype": "bf16"},
        # one decoding step of four prompts in four layers and the LM head of the 1.4 B generation benchmark model
        {"name": "decode_1.4B_4rows", "kind": "decode", "L": 4, "C": 2048, "NH": 32, "NKV": 8, "B": 4, "pos": 160, "max_len": 192},
        # one decoding step of 32 rows in LLaMA-3 8B layers with a long cache
        {"name": "decode_8B_32rows", "kind": "decode", "L": 4, "C": 4096, "NH": 32, "NKV": 8, "B": 32, "pos": 2000, "max_len": 2048},
        # prefill of one prompt of ordinary, odd length
        {"name": "prefill_1.4B_777", "kind": "prefill", "L": 4, "C": 2048, "NH": 32, "NKV": 8, "B": 1, "T": 777, "max_len": 1024},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention", "attention", "gqa", "mlp", "swiglu", "norm", "head", "update", "step", "decode", "decode", "prefill"])
    if kind == "attention":
        # 12x64 / 16x64 / 25x64: GPT-2; 16x96, 16x128, 32x80: GPT-3
        NH, HS = rng.choice([(12, 64), (16, 64), (25, 64), (16, 96), (16, 128), (32, 80)])
        T = rng.choice([64, 256, 512, 1024, 2048, _log(rng, 60, 2048), _log(rng, 60, 2048)])
        B = _log(rng, 1, max(1, min(64, 50_000_000 // (T * NH * HS))))
        return {"kind": kind, "B": B, "T": T, "NH": NH, "HS": HS}
    if kind == "gqa":
        NH, NKV, HS = rng.choice([(32, 8, 128), (32, 8, 64), (24, 8, 128)])
        T = rng.choice([512, 1024, 2048, 4096, _log(rng, 128, 4096)])
        return {"kind": kind, "B": _log(rng, 1, max(1, 8192 // T)), "T": T, "NH": NH, "NKV": NKV, "HS": HS}
    if kind == "mlp":
        C = rng.choice([384, 768, 1024, 1280, 1600])
        return {"kind": kind, "N": _log(rng, 256, 65536 * 768 * 768 // (C * C)), "C": C, "accumulate": rng.random() < 0.5}
    if kind == "swiglu":
        C, H = rng.choice([(2048, 8192), (3072, 8192), (4096, 14336)])
        return {"kind": kind, "N": _log(rng, 256, 4096), "C": C, "H": H, "accumulate": rng.random() < 0.5}
    if kind == "norm":
        rms = rng.random() < 0.4
        C = rng.choice([2048, 3072, 4096] if rms else [384, 768, 1024, 1280, 1600])
        return {"kind": kind, "N": _log(rng, 256, 65536 * 768 // C), "C": C, "rms": rms}
    if kind == "head":
        return {"kind": kind, "N": _log(rng, 256, 12000), "C": rng.choice([384, 768, 1024]), "V": 50257, "Vp": 50304}
    if kind == "update":
        return {"kind": kind, "depth": rng.choice([6, 12, 24])}
    if kind == "step":
        T = rng.choice([64, 128, 256, _log(rng, 60, 300)])
        return {"kind": kind, "depth": rng.choice([6, 12]), "B": _log(rng, 1, 8), "T": T, "dtype": "fp32" if rng.random() < 0.25 else "bf16"}
    L, C, NH, NKV = rng.choice([(4, 2048, 32, 8), (2, 2048, 32, 8), (2, 4096, 32, 8)])
    if kind == "decode":
        B, pos = _log(rng, 1, 32), _log(rng, 16, 2000)
        return {"kind": kind, "L": L, "C": C, "NH": NH, "NKV": NKV, "B": B, "pos": pos, "max_len": pos + 48}
    T = _log(rng, 16, 1024)
    return {"kind": kind, "L": L, "C": C, "NH": NH, "NKV": NKV, "B": _log(rng, 1, 4), "T": T, "max_len": T + 64}


# ---------------------------------------------------------------------------------------------------------------- inputs

class _Draw:
    """Tensors from one seeded generator on the GPU, in call order."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(seed)

    def n(self, *shape, std=1.0, mean=0.0, dtype=BF16):
        t = torch.randn(*shape, generator=self.g, device=DEV, dtype=F32 if math.prod(shape) < (1 << 24) else dtype)
        return (t * std + mean).to(dtype) if mean else t.mul_(std).to(dtype)

    def ids(self, hi, *shape):
        return torch.randint(0, hi, shape, generator=self.g, device=DEV, dtype=torch.int32)


def _rope(T, HS, theta=500000.0):
    """(T, HS/2, 2) cos / sin table of the rotary embedding."""
    f = 1.0 / (theta ** (torch.arange(0, HS, 2, dtype=F32) / HS))
    a = torch.outer(torch.arange(T, dtype=F32), f)
    return torch.stack([torch.cos(a), torch.sin(a)], dim=-1).contiguous().to(DEV)


def _empty(*shape, dtype=BF16):
    return torch.empty(*shape, dtype=dtype, device=DEV)


def _inputs(case, seed):
    """What both ``prepare`` and ``exact`` start from."""
    d, k, c = _Draw(seed), case["kind"], case
    if k == "attention":
        B, T, C = c["B"], c["T"], c["NH"] * c["HS"]
        return dict(qkv=d.n(B, T, 3 * C), dout=d.n(B, T, C))
    if k == "gqa":
        N, NH, NKV, HS = c["B"] * c["T"], c["NH"], c["NKV"], c["HS"]
        return dict(raw=d.n(N, (NH + 2 * NKV) * HS), dout=d.n(N, NH * HS), freqs=_rope(c["T"], HS))
    if k == "mlp":
        N, C = c["N"], c["C"]
        i = dict(x=d.n(N, C), w1=d.n(4 * C, C, std=0.02), b1=d.n(4 * C, std=0.02), w2=d.n(C, 4 * C, std=0.02), b2=d.n(C, std=0.02), dy=d.n(N, C))
        i.update(dw1=d.n(4 * C, C), dw2=d.n(C, 4 * C), db1=d.n(4 * C), db2=d.n(C))
        return i
    if k == "swiglu":
        N, C, H = c["N"], c["C"], c["H"]
        return dict(x=d.n(N, C), w12=d.n(2 * H, C, std=0.02), w3=d.n(C, H, std=0.02), dy=d.n(N, C), dw12=d.n(2 * H, C), dw3=d.n(C, H))
    if k == "norm":
        N, C = c["N"], c["C"]
        return dict(a=d.n(N, C), b=d.n(N, C), w=d.n(C, std=0.1, mean=1.0), bias=d.n(C, std=0.1), dy=d.n(N, C), dres=d.n(N, C),
                    dw=d.n(C), dbias=d.n(C), dcol=d.n(C))
    if k == "head":
        N, C, V, Vp = c["N"], c["C"], c["V"], c["Vp"]
        wte = d.n(Vp, C, std=0.02)
        wte[V:] = 0
        return dict(x=d.n(N, C), wte=wte, targets=d.ids(V, N))
    raise ValueError(k)


def _gpt_model(c, seed):
    from llmc_b200.models import gpt2
    dt = F32 if c.get("dtype") == "fp32" else BF16
    m = gpt2.GPT(gpt2.gpt2_descriptor(c["depth"]), DEV, dt, recompute=0)
    d = _Draw(seed)
    m.params_flat.copy_(d.n(m.num_parameters, std=0.02, dtype=dt))
    for n in ("ln1w", "ln2w", "lnfw"):
        m.params[n].add_(1.0)
    m.params["wte"][m.cfg.vocab_size:] = 0
    return m, d


def _llama_model(c, seed):
    from llmc_b200.models import llama3
    cfg = llama3.config_from_descriptor("llama3:l=%d,c=%d,h=%d,kv=%d,t=%d" % (c["L"], c["C"], c["NH"], c["NKV"], 2 * 2048))
    m = llama3.Llama(cfg, DEV, BF16, recompute=1)
    d = _Draw(seed)
    m.params_flat.copy_(d.n(m.num_parameters, std=0.02))
    for n in ("ln1w", "ln2w", "lnfw"):
        m.params[n].add_(1.0)
    return m, d


def prepare(case, seed):
    k, c = case["kind"], case
    if k == "step":
        if c["dtype"] == "fp32":
            torch.backends.cuda.matmul.allow_tf32 = True        # the trainer's default for the full-precision mode
        m, d = _gpt_model(c, seed)
        tok = d.ids(m.cfg.vocab_size, c["B"], c["T"] + 1)
        return dict(kind=k, m=m, x=tok[:, :-1].contiguous(), y=tok[:, 1:].contiguous())
    if k == "update":
        from llmc_b200.parallel.dist import DistConfig
        from llmc_b200.parallel.zero import ShardedAdamW
        m, d = _gpt_model(c, seed)
        opt = ShardedAdamW(m, DistConfig(0, 1, 0, torch.device(DEV, 0)), 0, True)
        m.allocate_grads()
        n = m.num_parameters
        m.grads_flat.copy_(d.n(n, std=1e-3))
        opt.m.copy_(d.n(n, std=1e-4, dtype=F32))
        opt.v.copy_(d.n(n, std=1e-3, dtype=F32).square_())
        opt.master.copy_(m.params_flat.float())
        opt.master_initialized = True
        return dict(kind=k, m=m, opt=opt, t=100)
    if k in ("decode", "prefill"):
        from llmc_b200.models import generate
        m, d = _llama_model(c, seed)
        dec = generate.CachedDecoder(m, c["B"], c["max_len"])
        if k == "prefill":
            return dict(kind=k, dec=dec, tokens=d.ids(m.cfg.vocab_size, c["B"], c["T"]))
        for l in range(c["L"]):
            dec.kcache[l, :, :c["pos"]] = d.n(c["B"], c["pos"], c["NKV"], c["C"] // c["NH"])
            dec.vcache[l, :, :c["pos"]] = d.n(c["B"], c["pos"], c["NKV"], c["C"] // c["NH"])
        tokens = d.ids(m.cfg.vocab_size, c["B"], 1)
        return dict(kind=k, step=generate.GraphStep(dec, c["B"], c["pos"]), pos=c["pos"], tokens=tokens, dec=dec)
    s = _inputs(case, seed)
    s["kind"] = k
    if k == "attention":
        B, T, NH = c["B"], c["T"], c["NH"]
        s.update(B=B, T=T, NH=NH, out=_empty(B, T, NH * c["HS"]), lse=_empty(B, NH, T, dtype=F32), dqkv=torch.empty_like(s["qkv"]))
    elif k == "gqa":
        B, T, NH, HS = c["B"], c["T"], c["NH"], c["HS"]
        N = B * T
        s.update(B=B, T=T, NH=NH, NKV=c["NKV"], packed=_empty(N, 3 * NH * HS), out=_empty(N, NH * HS), lse=_empty(B, NH, T, dtype=F32),
                 dpacked=_empty(N, 3 * NH * HS), draw=torch.empty_like(s["raw"]))
    elif k == "mlp":
        N, C = c["N"], c["C"]
        s.update(acc=c["accumulate"], pre=_empty(N, 4 * C), h=_empty(N, 4 * C), out=_empty(N, C), dpre=_empty(N, 4 * C), dx=_empty(N, C))
    elif k == "swiglu":
        N, C, H = c["N"], c["C"], c["H"]
        s.update(acc=c["accumulate"], x12=_empty(N, 2 * H), h=_empty(N, H), out=_empty(N, C), dh=_empty(N, H), dx12=_empty(N, 2 * H), dx=_empty(N, C))
    elif k == "norm":
        N, C = c["N"], c["C"]
        s.update(rms=c["rms"], res=_empty(N, C), out=_empty(N, C), mean=_empty(N, dtype=F32), rstd=_empty(N, dtype=F32))
    elif k == "head":
        N, C, V, Vp = c["N"], c["C"], c["V"], c["Vp"]
        s.update(V=V, logits=_empty(N, Vp), losses=torch.zeros(N, dtype=F32, device=DEV), dx=_empty(N, C), dw=_empty(Vp, C))
    return s


def run(s):
    from llmc_b200 import ops
    k = s["kind"]
    if k == "attention":
        ops.attention_forward(s["out"], s["lse"], s["qkv"], s["B"], s["T"], s["NH"])
        ops.attention_backward(s["dqkv"], s["dout"], s["qkv"], s["out"], s["lse"], s["B"], s["T"], s["NH"])
        return {n: s[n] for n in ("out", "lse", "dqkv")}
    if k == "gqa":
        B, T, NH, NKV = s["B"], s["T"], s["NH"], s["NKV"]
        ops.rope_forward(s["packed"], s["raw"], s["freqs"], T, NH, NKV)
        ops.attention_forward(s["out"], s["lse"], s["packed"], B, T, NH)
        ops.attention_backward(s["dpacked"], s["dout"], s["packed"], s["out"], s["lse"], B, T, NH)
        ops.rope_backward(s["draw"], s["dpacked"], s["freqs"], T, NH, NKV)
        return {n: s[n] for n in ("out", "lse", "draw")}
    if k == "mlp":
        acc = s["acc"]
        ops.matmul_forward(s["h"], s["x"], s["w1"], s["b1"], pre_gelu=s["pre"])
        ops.matmul_forward(s["out"], s["h"], s["w2"], s["b2"])
        ops.matmul_dgrad(s["dpre"], s["dy"], s["w2"], pre_gelu=s["pre"])
        ops.matmul_wgrad(s["dw2"], s["dy"], s["h"], accumulate=acc)
        ops.bias_grad(s["db2"], s["dy"], accumulate=acc)
        ops.bias_grad(s["db1"], s["dpre"], accumulate=acc)
        ops.matmul_dgrad(s["dx"], s["dpre"], s["w1"])
        ops.matmul_wgrad(s["dw1"], s["dpre"], s["x"], accumulate=acc)
        return {n: s[n] for n in ("out", "dx", "dw1", "dw2", "db1", "db2")}
    if k == "swiglu":
        acc = s["acc"]
        ops.matmul_forward(s["x12"], s["x"], s["w12"], None)
        ops.swiglu_forward(s["h"], s["x12"])
        ops.matmul_forward(s["out"], s["h"], s["w3"], None)
        ops.matmul_dgrad(s["dh"], s["dy"], s["w3"])
        ops.matmul_wgrad(s["dw3"], s["dy"], s["h"], accumulate=acc)
        ops.swiglu_backward(s["dx12"], s["dh"], s["x12"])
        ops.matmul_dgrad(s["dx"], s["dx12"], s["w12"])
        ops.matmul_wgrad(s["dw12"], s["dx12"], s["x"], accumulate=acc)
        return {n: s[n] for n in ("out", "dx", "dw12", "dw3")}
    if k == "norm":
        if s["rms"]:
            ops.rmsnorm_fused_residual_forward(s["res"], s["out"], s["rstd"], s["a"], s["b"], s["w"])
            ops.rmsnorm_backward(s["dres"], s["dw"], s["dy"], s["res"], s["w"], s["rstd"], accumulate_dinp=True, accumulate_dw=False)
            return {n: s[n] for n in ("res", "out", "rstd", "dres", "dw")}
        ops.fused_residual_forward(s["res"], s["out"], s["mean"], s["rstd"], s["a"], s["b"], s["w"], s["bias"])
        ops.layernorm_backward(s["dres"], s["dw"], s["dbias"], s["dy"], s["res"], s["w"], s["mean"], s["rstd"], accumulate_dinp=True,
                               accumulate_dwdb=False, dcolsum=s["dcol"], accumulate_dcol=False)
        return {n: s[n] for n in ("res", "out", "mean", "rstd", "dres", "dw", "dbias", "dcol")}
    if k == "head":
        ops.matmul_forward(s["logits"], s["x"], s["wte"], None)
        ops.fused_classifier(s["logits"], s["losses"], s["targets"], 1.0 / s["x"].shape[0], s["V"])
        ops.matmul_dgrad(s["dx"], s["logits"], s["wte"])
        ops.matmul_wgrad(s["dw"], s["logits"], s["x"], accumulate=False)
        return {"losses": s["losses"], "dlogits": s["logits"], "dx": s["dx"], "dw": s["dw"]}
    if k == "update":
        m, opt = s["m"], s["opt"]
        norm_sq = opt.grad_norm_sq()
        opt.step(1e-4, 0.1, s["t"])
        s["t"] += 1
        return {"params": m.params_flat, "master": opt.master, "m": opt.m, "v": opt.v, "norm_sq": norm_sq}
    if k == "step":
        m = s["m"]
        m.forward(s["x"], s["y"])
        m.backward()
        return {"loss": m.loss(), "losses": m.acts["losses"], "dlogits": m.acts["logits"], "grads": m.grads}
    if k == "decode":
        s["step"].pos.fill_(s["pos"])
        return s["step"].step(s["tokens"])
    if k == "prefill":
        dec = s["dec"]
        T = s["tokens"].shape[1]
        logits = dec.forward(s["tokens"], 0)
        return {"logits": logits, "k": dec.kcache[:, :, :T], "v": dec.vcache[:, :, :T]}
    raise ValueError(k)


# ---------------------------------------------------------------------------------------------------------------- float64 restatement

GELU_K = math.sqrt(2.0 / math.pi)


def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(GELU_K * (x + 0.044715 * x ** 3)))


def _attend(q, k, v):
    """Causal attention (B, T, NH, HS) -> out, lse (B, NH, T)."""
    T = q.shape[1]
    s = torch.einsum("bthd,bshd->bhts", q, k) * (1.0 / math.sqrt(q.shape[-1]))
    s = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device=q.device).triu(1), -math.inf)
    lse = torch.logsumexp(s, -1)
    return torch.einsum("bhts,bshd->bthd", torch.exp(s - lse.unsqueeze(-1)), v), lse


def _rotate(x, freqs):
    """x (..., T, heads, HS) rotated pairwise; freqs (T, HS/2, 2)."""
    c, s = freqs[..., 0].to(x.dtype).unsqueeze(-2), freqs[..., 1].to(x.dtype).unsqueeze(-2)
    re, im = x[..., 0::2], x[..., 1::2]
    return torch.stack([re * c - im * s, re * s + im * c], dim=-1).flatten(-2)


def _exact_attention(c, i):
    NH, HS, B, T = c["NH"], c["HS"], c["B"], c["T"]
    NKV = c.get("NKV")
    src = (i["qkv"].view(B, T, 3 * NH, HS) if NKV is None else i["raw"].view(B, T, NH + 2 * NKV, HS))
    dout = i["dout"].view(B, T, NH, HS)
    out, lse, dsrc = _empty(B, T, NH, HS, dtype=F64), _empty(B, NH, T, dtype=F64), _empty(*src.shape, dtype=F64)
    kv, rep = (NH, 1) if NKV is None else (NKV, NH // NKV)
    for b in range(B):
        for h in range(0, kv):
            qs, rows = slice(h * rep, (h + 1) * rep), [slice(h * rep, (h + 1) * rep), slice(NH + h, NH + h + 1), slice(NH + kv + h, NH + kv + h + 1)]
            q, k, v = (src[b:b + 1, :, r].double().requires_grad_(True) for r in rows)
            qr, kr = (q, k) if NKV is None else (_rotate(q, i["freqs"]), _rotate(k, i["freqs"]))
            o, l = _attend(qr, kr.expand(-1, -1, rep, -1), v.expand(-1, -1, rep, -1))
            for r, g in zip(rows, torch.autograd.grad(o, (q, k, v), dout[b:b + 1, :, qs].double())):
                dsrc[b:b + 1, :, r] = g
            out[b:b + 1, :, qs], lse[b:b + 1, qs] = o.detach(), l.detach()
    if NKV is None:
        return {"out": out.view(B, T, NH * HS), "lse": lse, "dqkv": dsrc.view(B, T, 3 * NH * HS)}
    return {"out": out.view(B * T, NH * HS), "lse": lse, "draw": dsrc.view(B * T, -1)}


def _exact_gpt(c, p, x, y, cfg):
    """Loss, per-token losses, dlogits and parameter gradients of GPT-2 in float64."""
    p = {n: t.double().requires_grad_(True) for n, t in p.items()}
    B, T = x.shape
    C, NH, V, Vp = cfg.channels, cfg.num_heads, cfg.vocab_size, cfg.padded_vocab_size
    ln = lambda h, w, b: torch.nn.functional.layer_norm(h, (C,), w, b, 1e-5)
    h = p["wte"][x.long()] + p["wpe"][:T]
    for l in range(cfg.num_layers):
        q, k, v = (ln(h, p["ln1w"][l], p["ln1b"][l]) @ p["qkvw"][l].t() + p["qkvb"][l]).view(B, T, 3, NH, C // NH).unbind(2)
        h = h + _attend(q, k, v)[0].reshape(B, T, C) @ p["attprojw"][l].t() + p["attprojb"][l]
        u = _gelu(ln(h, p["ln2w"][l], p["ln2b"][l]) @ p["fcw"][l].t() + p["fcb"][l])
        h = h + u @ p["fcprojw"][l].t() + p["fcprojb"][l]
    logits = (ln(h, p["lnfw"], p["lnfb"]) @ p["wte"].t()).view(B * T, Vp)
    logits.retain_grad()
    losses = torch.nn.functional.cross_entropy(logits[:, :V], y.long().view(-1), reduction="none")
    losses.mean().backward()
    return {"loss": losses.detach().mean(), "losses": losses.detach(), "dlogits": logits.grad, "grads": {n: t.grad for n, t in p.items()}}


def _exact_llama(m, tokens, start, kc, vc):
    """Logits of the last position and the layers' new keys / values, float64; kc / vc: cached keys and values (L, B, S, NKV, HS) or None."""
    cfg, p = m.cfg, m.params
    B, T = tokens.shape
    NH, NKV, HS, C, H = cfg.num_heads, cfg.num_kv_heads, cfg.head_size, cfg.channels, cfg.hidden_dim
    rms = lambda h, w: h * torch.rsqrt(h.square().mean(-1, keepdim=True) + cfg.norm_eps) * w.double()
    freqs = _rope_scaled(start + T, HS)[start:]
    x = p["wte"][tokens.long()].double()
    ks, vs = [], []
    for l in range(cfg.num_layers):
        raw = (rms(x, p["ln1w"][l]) @ p["qkvw"][l].double().t()).view(B, T, NH + 2 * NKV, HS)
        q, k, v = _rotate(raw[:, :, :NH], freqs), _rotate(raw[:, :, NH:NH + NKV], freqs), raw[:, :, NH + NKV:]
        ks.append(k)
        vs.append(v)
        if kc is not None:
            k, v = torch.cat([kc[l].double(), k], 1), torch.cat([vc[l].double(), v], 1)
        s = torch.einsum("btgrd,bsgd->bgrts", q.view(B, T, NKV, NH // NKV, HS), k) / math.sqrt(HS)
        s = s.masked_fill(torch.ones(T, start + T, dtype=torch.bool, device=DEV).triu(start + 1), -math.inf)
        a = torch.einsum("bgrts,bsgd->btgrd", torch.softmax(s, -1), v).reshape(B, T, C)
        x = x + a @ p["attprojw"][l].double().t()
        u = rms(x, p["ln2w"][l]) @ p["fc12w"][l].double().t()
        x = x + (u[..., :H] * torch.nn.functional.silu(u[..., H:])) @ p["fcprojw"][l].double().t()
    logits = rms(x[:, -1], p["lnfw"]) @ p["lmhead"].double().t()
    return logits[:, :cfg.vocab_size], torch.stack(ks), torch.stack(vs)


def _rope_scaled(T, HS):
    """The LLaMA-3.1 table: low frequencies divided by 8, a smooth transition between wavelengths 2048 and 8192."""
    f = 1.0 / (500000.0 ** (torch.arange(0, HS, 2, dtype=F32) / HS))
    w = 2 * math.pi / f
    s = ((8192 / w - 1) / 3).clamp(0, 1)
    f = (1 - s) * f / 8 + s * f
    a = torch.outer(torch.arange(T, dtype=F32), f)
    return torch.stack([torch.cos(a), torch.sin(a)], dim=-1).to(DEV)


def exact(case, seed):
    k, c = case["kind"], case
    if k == "step":
        s = prepare(case, seed)
        return _exact_gpt(c, s["m"].params, s["x"], s["y"], s["m"].cfg)
    if k == "update":
        s = prepare(case, seed)
        opt, t, lr, wd = s["opt"], s["t"], 1e-4, 0.1
        g = s["m"].grads_flat.double()
        norm_sq = g.square().sum()
        g *= min(1.0, opt.grad_clip / math.sqrt(float(norm_sq)))
        mm = opt.m.double() * opt.beta1 + g * (1 - opt.beta1)
        vv = opt.v.double() * opt.beta2 + g.square() * (1 - opt.beta2)
        old = opt.master.double()
        decay = torch.zeros(old.numel(), dtype=torch.bool, device=DEV)
        for n, off, per, L in s["m"].tensor_sizes():
            decay[off:off + per * L] = n in ("wte", "wpe", "qkvw", "attprojw", "fcw", "fcprojw")
        new = old - lr * ((mm / (1 - opt.beta1 ** t)) / (torch.sqrt(vv / (1 - opt.beta2 ** t)) + opt.eps) + wd * decay * old)
        # the bf16 parameters are rounded stochastically: no exact value
        return {"params": None, "master": new, "m": mm, "v": vv, "norm_sq": norm_sq.view(1)}
    if k in ("decode", "prefill"):
        if k == "prefill":
            s = prepare(case, seed)
            logits, kk, vv = _exact_llama(s["dec"].model, s["tokens"], 0, None, None)
            return {"logits": logits, "k": kk, "v": vv}
        s = prepare(case, seed)
        dec, pos = s["dec"], s["pos"]
        return _exact_llama(dec.model, s["tokens"], pos, dec.kcache[:, :, :pos], dec.vcache[:, :, :pos])[0]
    i = _inputs(case, seed)
    if k in ("attention", "gqa"):
        return _exact_attention(c, i)
    i = {n: t.double() if t.is_floating_point() else t for n, t in i.items()}
    if k == "mlp":
        a = 1.0 if c["accumulate"] else 0.0
        pre = i["x"] @ i["w1"].t() + i["b1"]
        th = torch.tanh(GELU_K * (pre + 0.044715 * pre ** 3))
        h = 0.5 * pre * (1 + th)
        dpre = (i["dy"] @ i["w2"]) * (0.5 * (1 + th) + 0.5 * pre * (1 - th * th) * GELU_K * (1 + 3 * 0.044715 * pre * pre))
        return {"out": h @ i["w2"].t() + i["b2"], "dx": dpre @ i["w1"], "dw1": a * i["dw1"] + dpre.t() @ i["x"], "dw2": a * i["dw2"] + i["dy"].t() @ h,
                "db1": a * i["db1"] + dpre.sum(0), "db2": a * i["db2"] + i["dy"].sum(0)}
    if k == "swiglu":
        a, H = 1.0 if c["accumulate"] else 0.0, c["H"]
        x12 = i["x"] @ i["w12"].t()
        x1, x2 = x12[:, :H], x12[:, H:]
        sg = torch.sigmoid(x2)
        h, dh = x1 * x2 * sg, i["dy"] @ i["w3"]
        dx12 = torch.cat([dh * x2 * sg, dh * x1 * sg * (1 + x2 * (1 - sg))], 1)
        return {"out": h @ i["w3"].t(), "dx": dx12 @ i["w12"], "dw12": a * i["dw12"] + dx12.t() @ i["x"], "dw3": a * i["dw3"] + i["dy"].t() @ h}
    if k == "norm":
        # the library normalises the bf16 sum that it stores, so that forward and backward see the same values
        res = i["a"] + i["b"]
        r = res.to(BF16).double()
        mean = torch.zeros_like(r[:, :1]) if c["rms"] else r.mean(-1, keepdim=True)
        rstd = torch.rsqrt((r - mean).square().mean(-1, keepdim=True) + 1e-5)
        n = (r - mean) * rstd
        dn = i["dy"] * i["w"]
        dx = dn - n * (dn * n).mean(-1, keepdim=True)
        dres = i["dres"] + (dx if c["rms"] else dx - dn.mean(-1, keepdim=True)) * rstd
        dw = (i["dy"] * n).sum(0)
        if c["rms"]:
            return {"res": res, "out": n * i["w"], "rstd": rstd.view(-1), "dres": dres, "dw": dw}
        return {"res": res, "out": n * i["w"] + i["bias"], "mean": mean.view(-1), "rstd": rstd.view(-1), "dres": dres, "dw": dw,
                "dbias": i["dy"].sum(0), "dcol": dres.sum(0)}
    if k == "head":
        V, N = c["V"], c["N"]
        logits = i["x"] @ i["wte"][:V].t()
        tgt = i["targets"].long()
        lse = torch.logsumexp(logits, -1)
        losses = lse - logits.gather(1, tgt.view(-1, 1)).view(-1)
        dlogits = torch.zeros(N, c["Vp"], dtype=F64, device=DEV)
        dlogits[:, :V] = torch.exp_(logits.sub_(lse.view(-1, 1)))
        dlogits[torch.arange(N, device=DEV), tgt] -= 1.0
        dlogits /= N
        return {"losses": losses, "dlogits": dlogits, "dx": dlogits @ i["wte"], "dw": dlogits.t() @ i["x"]}
    raise ValueError(k)


# ---------------------------------------------------------------------------------------------------------------- work and tolerance

def work(case):
    k, c = case["kind"], case
    if k in ("attention", "gqa"):
        B, T, NH, HS = c["B"], c["T"], c["NH"], c["HS"]
        N, src = B * T, (3 * NH if k == "attention" else NH + 2 * c["NKV"]) * HS
        # qkv, dout in; out, lse, dqkv out; two causal products forward, five backward
        return {"bytes": 2.0 * N * (2 * src + 2 * NH * HS) + 4.0 * N * NH, "flops": 7.0 * B * NH * T * T * HS}
    if k == "mlp":
        N, C, a = c["N"], c["C"], 2 if c["accumulate"] else 1
        return {"bytes": 2.0 * (4 * N * C + 8 * C * C * (1 + a) + 5 * C * (1 + a)), "flops": 48.0 * N * C * C}
    if k == "swiglu":
        N, C, H, a = c["N"], c["C"], c["H"], 2 if c["accumulate"] else 1
        return {"bytes": 2.0 * (4 * N * C + 3 * C * H * (1 + a)), "flops": 18.0 * N * C * H}
    if k == "norm":
        N, C = c["N"], c["C"]
        return {"bytes": 2.0 * 7 * N * C + 8.0 * N, "flops": 30.0 * N * C}        # a, b, dy, dres in; res, out, dres out
    if k == "head":
        N, C, Vp = c["N"], c["C"], c["Vp"]
        return {"bytes": 2.0 * (2 * N * C + 2 * Vp * C + N * Vp) + 8.0 * N, "flops": 6.0 * N * C * Vp}
    if k == "update":
        n = _gpt_size(c["depth"])[0]
        return {"bytes": n * (2.0 + 2.0 + 24.0), "flops": 15.0 * n}               # gradients in, parameters out, master / m / v both ways
    if k == "step":
        n, L, C = _gpt_size(c["depth"])
        N, e = c["B"] * c["T"], 4 if c["dtype"] == "fp32" else 2
        return {"bytes": float(e) * (2 * n + N * 50304), "flops": 6.0 * n * N + 7.0 * L * C * N * c["T"]}
    L, C, NH, NKV, B = c["L"], c["C"], c["NH"], c["NKV"], c["B"]
    HS = C // NH
    H = 1024 * ((int(1.3 * int(8 * C / 3)) + 1023) // 1024)
    layer, head = (NH + 2 * NKV) * HS * C + C * C + 3 * H * C, 128256 * C
    if k == "decode":
        return {"bytes": 2.0 * (L * layer + head) + 4.0 * L * B * c["pos"] * NKV * HS + 4.0 * B * 128256,
                "flops": 2.0 * B * (L * layer + head) + 4.0 * L * B * c["pos"] * C}
    N = B * c["T"]
    return {"bytes": 2.0 * (L * layer + head) + 4.0 * L * N * NKV * HS + 4.0 * B * 128256,
            "flops": 2.0 * N * L * layer + 2.0 * B * head + 2.0 * L * B * c["T"] * c["T"] * C}


def _gpt_size(depth):
    C = {6: 384, 12: 768, 24: 1024}[depth]
    return 50304 * C + 1024 * C + depth * (12 * C * C + 13 * C) + 2 * C, depth, C


def tolerance(case):
    """Relative errors of results that are rounded to bf16 once or twice on the way (half an ulp is 2^-9 = 0.002), measured against ``exact``;
    ``max`` covers single elements of small gradients and sums of many rounded terms."""
    k = case["kind"]
    if k == "update":
        return {"rel": 1e-4, "max": 2e-2}          # fp32 state; a bf16 parameter may round to the other neighbour
    if k in ("decode", "prefill"):
        return {"rel": 3e-2, "max": 0.5}           # roundings of several layers: 0.016 against exact on either side
    if k == "step":
        return {"rel": 3e-2, "max": 0.9}           # 0.011 on the gradients of twelve layers
    return {"rel": 1e-2, "max": 0.3}
