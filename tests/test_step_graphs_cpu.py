"""When a micro-step may be replayed: every buffer that its launches read or write is the one they were captured with."""
import contextlib
import copy
import gc
import pickle
import threading
from types import SimpleNamespace

import pytest
import torch

from llmc_b200.models import gpt2, step_graphs
from llmc_b200.ops import kernels as KN


def fake_model():
    z = lambda: torch.zeros(4)
    return SimpleNamespace(device=SimpleNamespace(type="cuda"), dtype=torch.bfloat16, use_graphs=True, params_flat=z(), params={"w": z()}, inputs=z(),
                           targets=z(), acts={"x": z()}, grads={"w": z()}, grads_flat=z(), freqs=z())


@pytest.mark.parametrize("name", ["params_flat", "params", "inputs", "targets", "acts", "grads", "grads_flat", "freqs"])
def test_a_replaced_buffer_is_launched_and_captured_again(monkeypatch, name):
    m, g, calls = fake_model(), step_graphs.StepGraphs(), []
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(step_graphs.StepGraphs, "_capture",
                        staticmethod(lambda model, e, fn: e.update(launches=0, graph=SimpleNamespace(replay=lambda: calls.append("replay")))))
    for _ in range(4):
        g.run(m, 64, ("forward",), lambda: calls.append("launch"))
    assert calls == ["launch", "launch", "replay", "replay"]
    old = getattr(m, name)                                     # stays alive: a new tensor cannot get its address
    setattr(m, name, {k: t.clone() for k, t in old.items()} if isinstance(old, dict) else old.clone())
    calls.clear()
    for _ in range(3):
        g.run(m, 64, ("forward",), lambda: calls.append("launch"))
    assert calls == ["launch", "launch", "replay"]


def test_a_capture_holds_the_scratch_buffers_it_took_and_no_others():
    dev = torch.device("cpu")
    try:
        other = KN._scratch.get("test_other", 1000, torch.float32, dev)
        with KN.scratch_taken() as outer:
            a = KN._scratch.get("test_a", 10, torch.float32, dev)
            with KN.scratch_taken() as inner:
                b = KN._scratch.get("test_a", 20, torch.float32, dev)          # outgrown inside: both are part of the capture
            assert len(inner) == 1 and inner[0] is b
        assert [id(t) for t in outer] == [id(a), id(b)]
        KN._scratch.get("test_a", 30, torch.float32, dev)
        assert len(outer) == 2 and all(t is not other for t in outer)
    finally:
        for k in [k for k in KN._scratch.bufs if k[0].startswith("test_")]:
            del KN._scratch.bufs[k]


def test_a_model_with_captured_steps_can_be_copied_and_pickled():
    m = gpt2.GPT(gpt2.GPTConfig(32, 100, 128, 1, 2, 64), "cpu", torch.float32)
    m.init_random(1)
    m.step_graphs._entries["forward"] = {"graph": (i for i in ())}             # like a CUDA graph, it can be neither copied nor pickled
    for c in (copy.deepcopy(m), pickle.loads(pickle.dumps(m))):
        assert torch.equal(c.params_flat, m.params_flat) and not c.step_graphs._entries
        tok = torch.arange(32, dtype=torch.int32).view(1, 32)
        c.forward(tok, tok)
        m.forward(tok, tok)
        assert torch.equal(c.loss(), m.loss())


@pytest.mark.parametrize("enabled", [True, False])
def test_no_collection_in_a_capture_while_another_thread_ends_its_own(monkeypatch, enabled):
    graph = SimpleNamespace(capture_begin=lambda capture_error_mode: None, capture_end=lambda: None)
    monkeypatch.setattr(torch.cuda, "CUDAGraph", lambda: graph)
    monkeypatch.setattr(torch.cuda, "Stream", lambda device: None)
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    both_inside, first_out, seen = threading.Barrier(2), threading.Event(), []

    def model():
        return SimpleNamespace(device=None, step_graphs=step_graphs.StepGraphs())

    def first():
        step_graphs.StepGraphs._capture(model(), {}, lambda: both_inside.wait(20))
        first_out.set()

    def second():
        def launches():
            both_inside.wait(20)
            first_out.wait(20)
            seen.append(gc.isenabled())
        step_graphs.StepGraphs._capture(model(), {}, launches)

    before = gc.isenabled()
    try:
        (gc.enable if enabled else gc.disable)()
        threads = [threading.Thread(target=f) for f in (first, second)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert seen == [False] and gc.isenabled() == enabled
    finally:
        (gc.enable if before else gc.disable)()


# tokens of a captured pass whose chain gets the priority: fewer for wide layers
@pytest.mark.parametrize("channels,tokens", [(64, 1536), (768, 1536), (1280, 1536), (1600, 1048), (2048, 640), (2560, 409), (4096, 160)])
def test_the_chain_comes_first_up_to(channels, tokens):
    with torch.device("meta"):
        m = gpt2.GPT(gpt2.GPTConfig(16, 100, 128, 1, channels // 64, channels), "meta", torch.bfloat16)
    assert m.chain_first_tokens == tokens
