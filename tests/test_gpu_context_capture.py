"""A context for the primitives alone allocates nothing that a caller's
global-mode stream capture refuses: it can be created during one, and the
captured work replays."""
import pytest

from qutree_gb300 import qtgpu

pytestmark = pytest.mark.gpu


def test_context_created_during_a_global_capture():
    import torch
    x = torch.zeros(1024, device="cuda")
    x += 1
    torch.cuda.synchronize()
    qtgpu.load()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="global"):
        x += 1
        ctx = qtgpu.Context(0)
    g.replay()
    torch.cuda.synchronize()
    assert float(x.sum()) == 2048.0
    ctx.sync()  # nothing prepared: a plain wait
    ctx.close()
