"""No garbage collection inside the capture of a micro-step: one that frees the graphs of a dropped model there invalidates the capture."""
import gc

import pytest
import torch

from llmc_b200.models import gpt2

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("enabled", [True, False])
def test_no_collection_during_capture(enabled):
    m = gpt2.GPT(gpt2.GPTConfig(64, 1000, 1024, 1, 2, 128), DEV, torch.bfloat16)
    m.init_random(3)
    tok = torch.randint(0, 500, (2, 65), dtype=torch.int32).to(DEV)
    x, y = tok[:, :-1].contiguous(), tok[:, 1:].contiguous()
    launch, seen = m._forward, []

    def forward(*args):
        seen.append((torch.cuda.is_current_stream_capturing(), gc.isenabled()))
        return launch(*args)

    m._forward = forward
    before = gc.isenabled()
    try:
        (gc.enable if enabled else gc.disable)()
        for _ in range(4):
            m.forward(x, y, 1, 0)
            assert gc.isenabled() == enabled
    finally:
        (gc.enable if before else gc.disable)()
    assert seen == [(False, enabled), (False, enabled), (True, False)]          # the fourth is a replay
    assert torch.isfinite(m.loss(1)).all()
