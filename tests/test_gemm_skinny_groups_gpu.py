"""The weight-streaming product when a block takes several groups of rows in turn: a launch of more groups than blocks run at a
time gives the bits of launches that hold a few of its groups each."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# 2 blocks an SM and more groups than that at 3; K of fewer chunks than warps, of fewer than stages, of several rounds, ragged
@pytest.mark.parametrize("N", [16 * 444, 16 * 444 + 16, 16 * 1000 + 8, 16 * 2000])
@pytest.mark.parametrize("K", [64, 136, 1024, 2056])
@pytest.mark.parametrize("M", [1, 5, 8])
def test_groups_in_turn(M, K, N):
    from lmsf_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(N + K + M)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).bfloat16()
    torch.cuda.synchronize()
    step = 16 * 100                                       # few enough groups for one round of blocks
    whole = torch.full((M, N), float("nan"), device="cuda")
    kernels.gemm_skinny(whole, x, w)
    for a in range(0, N, step):
        part = torch.empty((M, min(step, N - a)), device="cuda")
        kernels.gemm_skinny(part, x, w[a:a + step])
        assert torch.equal(part, whole[:, a:a + step]), a
    # gated: rows of the two halves side by side
    half = N // 2 // 8 * 8
    gated = torch.full((M, half), float("nan"), device="cuda")
    sumsq = torch.rand(M, 8, device="cuda", generator=g)[:, :5]
    both = w[:2 * half].contiguous()
    kernels.gemm_skinny(gated, x, both, fuse_act="silu", prenorm=(sumsq, 1e-5, K))
    for a in range(0, half, 800):
        rows = torch.cat([both[a:min(a + 800, half)], both[half + a:half + min(a + 800, half)]]).contiguous()
        part = torch.empty((M, rows.shape[0] // 2), device="cuda")
        kernels.gemm_skinny(part, x, rows, fuse_act="silu", prenorm=(sumsq, 1e-5, K))
        assert torch.equal(part, gated[:, a:a + 800]), a
    # residual form
    res, nw = torch.randn(M, N, device="cuda", generator=g), torch.rand(N, device="cuda", generator=g) + 0.5
    parts = kernels.gemm_skinny_residual_parts(N)
    sums = torch.full((M, (parts + 3) // 4 * 4), float("nan"), device="cuda")[:, :parts]
    out, want = torch.empty(M, N, device="cuda", dtype=torch.bfloat16), res + whole.bfloat16().float()
    kernels.gemm_skinny_residual(out, x, w, res, nw, sums)
    assert torch.equal(res, want) and torch.equal(out, (want * nw).bfloat16())
    squares = torch.nn.functional.pad(want.double().square(), (0, parts * 16 - N)).view(M, parts, 16).sum(-1)
    assert torch.allclose(sums.double(), squares, rtol=16 * 2.0 ** -24, atol=0)
