"""The branches of a captured backward pass (models/step_graphs.py, Side): every two launches that touch the same memory, one of them to write it, follow one
another.  The operators only note what they read and write; streams and events are clocks, so that a missing join shows without running anything."""
import contextlib
import types

import pytest
import torch
import torch.overrides

from llmc_b200.models import gpt2, llama3, step_graphs


class Stream:
    def __init__(self, world):
        self.world, self.clock = world, {}

    def tick(self):
        self.clock[self] = self.clock.get(self, 0) + 1
        return self.clock[self]

    def record_event(self):
        return dict(self.clock)

    def wait_event(self, event):
        if self is self.world.main and all(self.clock.get(s, 0) >= n for s, n in event.items()):
            self.world.idle_waits += 1
        for s, n in event.items():
            self.clock[s] = max(self.clock.get(s, 0), n)


class World:
    """Stands for both ``ops`` and ``torch.cuda``."""

    def __init__(self):
        self.main = Stream(self)
        self.now = self.main
        self.log, self.scratch, self.idle_waits = [], {}, 0

    # ---- torch.cuda
    def current_stream(self):
        return self.now

    @contextlib.contextmanager
    def stream(self, s):
        before, self.now = self.now, s
        yield
        self.now = before

    # ---- launches
    def launch(self, name, writes, reads):
        n = self.now.tick()
        for t, write in [(t, True) for t in writes] + [(t, False) for t in reads]:
            if t is None:
                continue
            lo, hi = t if isinstance(t, tuple) else (t.data_ptr(), t.data_ptr() + t.numel() * t.element_size())
            for other, s, m, a, b, w in self.log:
                if lo < b and a < hi and (write or w) and s is not self.now:
                    assert self.now.clock.get(s, 0) >= m, "%s does not follow %s" % (name, other)
            self.log.append((name, self.now, n, lo, hi, write))

    def own(self, name):
        i = self.scratch.setdefault(name, len(self.scratch))
        return (-2 * i - 2, -2 * i - 1)

    def __getattr__(self, name):
        def op(out, *args, **kw):
            tensors = [t for t in args if torch.is_tensor(t)]
            if name in ("layernorm_backward", "rmsnorm_backward"):
                n = 2 if name == "layernorm_backward" else 1
                part = self.own("norm sums")
                self.launch(name, [out, part], tensors[n:] + [kw.get("dinp_old", out)])
                with (kw.get("sums_in") or contextlib.nullcontext)():
                    self.launch(name + " sums", tensors[:n] + [kw.get("dcolsum")], [part])
                return
            writes = [out] + ([self.own(name)] if name in ("matmul_wgrad", "bias_grad", "attention_backward") else [])
            if name in ("layernorm_forward", "rmsnorm_forward"):
                tensors = [t for t in tensors if t is not None]
            if name == "encoder_backward":
                writes += [tensors.pop(0)] if torch.is_tensor(args[0]) else []
            self.launch(name, writes, tensors + [kw.get("pre_gelu")])
        return op


def _model(family, recompute):
    if family == "gpt2":
        m = gpt2.GPT(gpt2.GPTConfig(16, 100, 128, 3, 2, 64), "cpu", torch.float32, recompute=recompute)
    else:
        m = llama3.Llama(llama3.config_from_descriptor("llama3:l=3,c=64,h=2,kv=1,t=16,v=100,m=64,f=1.0"), "cpu", torch.float32, recompute=recompute)
    m.allocate_grads()
    m.forward(torch.zeros(2, 16, dtype=torch.int32), torch.zeros(2, 16, dtype=torch.int32))
    return m


def _run(monkeypatch, family, recompute, spoil=None):
    m, world = _model(family, recompute), World()
    monkeypatch.setattr(gpt2 if family == "gpt2" else llama3, "ops", world)
    fake = types.SimpleNamespace(cuda=world, empty_like=torch.empty_like)
    monkeypatch.setattr(step_graphs, "torch", fake)
    side = step_graphs.Side(Stream(world), Stream(world))
    if spoil:
        monkeypatch.setattr(side, spoil, lambda *a: None)
    m.step_graphs.side = side
    m._backward(2, 16, 0, None)
    # the graph ends with the main branch: it has to follow everything
    assert all(world.main.clock.get(s, 0) >= s.clock.get(s, 0) for s in (side.stream, side.sums))
    return world


@pytest.mark.parametrize("recompute", [0, 1, 2])
@pytest.mark.parametrize("family", ["gpt2", "llama3"])
def test_launches_on_the_same_memory_follow_one_another(monkeypatch, family, recompute):
    world = _run(monkeypatch, family, recompute)
    assert len({s for _, s, *_ in world.log}) == (3 if family == "gpt2" else 2)
    # and none of the chain waits for what it follows already: a launch with an edge from another branch does not start under the one before it
    assert world.idle_waits == 0


@pytest.mark.parametrize("family", ["gpt2", "llama3"])
def test_a_missing_join_is_found(monkeypatch, family):
    with pytest.raises(AssertionError, match="does not follow"):
        _run(monkeypatch, family, 0, spoil="free")


class Views(torch.overrides.TorchFunctionMode):
    """The views t[i] taken."""

    def __init__(self):
        super().__init__()
        self.taken = []

    def __torch_function__(self, func, types, args=(), kwargs=None):
        if func is torch.Tensor.__getitem__:
            self.taken.append((args[0].data_ptr(), args[0].shape, args[1]))
        return func(*args, **(kwargs or {}))


# Outside a capture a pass of a small batch is bound by the host, and a view takes it longer than a launch takes the GPU: what a buffer's readers and writers are told
# apart by must not be viewed again (4 x 64 tokens of GPT-2 124M 4.62 ms, 4.74 with three more views a layer)
@pytest.mark.parametrize("family,passes", [("gpt2", ("_forward", "_backward")), ("llama3", ("_backward",))])
def test_each_layer_of_a_buffer_is_viewed_once(monkeypatch, family, passes):
    m = _model(family, 0)
    monkeypatch.setattr(gpt2 if family == "gpt2" else llama3, "ops", World())
    for name in passes:
        with Views() as views:
            m._backward(2, 16, 0, None) if name == "_backward" else m._forward(2, 16, None, False, False)
        assert len(views.taken) > 3 * m.cfg.num_layers and len(views.taken) == len({repr(v) for v in views.taken}), name
