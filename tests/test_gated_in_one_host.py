"""When a feed-forward's gate, up and activation run as one kernel: the choice, without a GPU."""
import pytest
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


# (width, features, rows): product and activation apart against the gated kernel, as measured with cold weights on a device of 148 SMs
SLOWER = [(4096, 14336, 300), (4096, 14336, 384), (4096, 14336, 560), (4096, 14336, 769), (4096, 14336, 829), (4096, 14336, 860), (4096, 14336, 1025),
          (5120, 13824, 240), (5120, 13824, 380), (5120, 13824, 420), (5120, 13824, 614), (5120, 13824, 680), (3072, 8192, 1040),
          (8192, 28672, 600), (8192, 28672, 1100), (8192, 28672, 1300), (4096, 11008, 850), (2048, 5632, 512), (2048, 8192, 330)]
FASTER = [(4096, 14336, 237), (4096, 14336, 256), (4096, 14336, 512), (4096, 14336, 600), (4096, 14336, 768), (4096, 14336, 1024), (4096, 14336, 1500),
          (4096, 14336, 2048), (4096, 14336, 8192), (5120, 13824, 512), (5120, 13824, 1024), (5120, 13824, 2048), (3072, 8192, 256), (3072, 8192, 1200),
          (8192, 28672, 512), (8192, 28672, 1500), (2048, 8192, 208), (2048, 8192, 860), (2048, 8192, 2048), (2048, 5632, 1000), (1024, 4096, 512),
          (512, 2048, 4096)]


@pytest.mark.parametrize("width,features,rows", SLOWER + FASTER)
def test_the_kernel_is_taken_where_it_was_measured_to_be_faster(width, features, rows, monkeypatch):
    """SLOWER: by 3 % and more; FASTER: by 4 % and more."""
    monkeypatch.setattr(kernels, "sm_count", lambda device: 148)
    assert linear.gated_in_one(rows, width, features, "cuda:0") == ((width, features, rows) in FASTER)
