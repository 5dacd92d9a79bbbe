"""When a micro-step may be replayed: every buffer that its launches read or write is the one they were captured with."""
from types import SimpleNamespace

import pytest
import torch

from llmc_b200.models import step_graphs


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

