"""When a feed-forward's gate, up and activation run as one kernel: the choice, without a GPU."""
import torch

from lmsf_b200 import kernels
from lmsf_b200.parts import linear
from lmsf_b200.parts.mlp import GatedMLP


def test_the_part_needs_no_step(monkeypatch):
    """A feed-forward called alone, with None for the step: the kernel is given no error word, and its face takes the device's."""
    seen = []

    def gated(out, x, w, act, error_flag=None):
        seen.append(error_flag)
        gate, up = (x.float() @ w.float().T).chunk(2, 1)
        out.copy_(torch.nn.functional.silu(gate) * up)

    monkeypatch.setattr(kernels, "gemm_gated_tc", gated)
    monkeypatch.setattr(linear, "gated_in_one", lambda *a: True)
    g = torch.Generator().manual_seed(3)
    part = GatedMLP(hidden_size=64, intermediate_size=96)
    w = {"gate_up": torch.randn((192, 64), generator=g).to(torch.bfloat16), "down": torch.randn((64, 96), generator=g).to(torch.bfloat16)}
    part.set_weights(w)
    x = torch.randn((40, 64), generator=g).to(torch.bfloat16)
    y = part.forward(None, x)
    assert seen == [None] and y.shape == (40, 64) and torch.isfinite(y).all()
