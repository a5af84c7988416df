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


# about 1,000 groups: a block goes from rotated to unrotated rows, from q to k, v and the rows behind them between its groups
@pytest.mark.parametrize("nh,nkv,hd,rot,neox,planes,extra", [(40, 40, 128, 128, True, 2, 0), (48, 40, 128, 64, True, 2, 0), (40, 40, 128, 32, False, 2, 0),
                                                            (100, 24, 112, 48, True, 1, 16 * 41), (70, 60, 80, 0, True, 1, 16 * 333)])
@pytest.mark.parametrize("M,K", [(1, 136), (5, 1024), (8, 2056)])
def test_groups_in_turn_with_rotation_and_cache_write(M, K, nh, nkv, hd, rot, neox, planes, extra):
    from lmsf_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(M + nh + rot)
    bs, n_pages, n_seqs = 8, 24, 3
    q_size, kv_size = nh * hd, nkv * hd
    N = q_size + planes * kv_size + extra
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g).bfloat16()
    sumsq = torch.rand(M, 8, device="cuda", generator=g)[:, :5]
    inv_freq = (10000.0 ** (-torch.arange(0, rot, 2, device="cuda").float() / rot)) if rot else None
    token_seq = torch.tensor([i % n_seqs for i in range(M)], dtype=torch.int32, device="cuda")
    positions = torch.tensor([(i // n_seqs) * 5 + (i % n_seqs) * 3 for i in range(M)], dtype=torch.int32, device="cuda")
    table = torch.randperm(n_pages, device="cuda", generator=g)[:n_seqs * 4].to(torch.int32).view(n_seqs, 4).contiguous()
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    for kw in ({}, {"bias": bias, "prenorm": (sumsq, 1e-5, K)}):
        # the product from launches of a few groups each, then the rotation and the cache write of their own
        p = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
        for a in range(0, N, 1600):
            rows = slice(a, min(a + 1600, N))
            kernels.gemm_skinny(p[:, rows], x, w[rows], **(dict(kw, bias=bias[rows].clone()) if kw else {}))
        want = torch.zeros(n_pages, planes, nkv, bs, hd, device="cuda", dtype=torch.bfloat16)
        kernels.rope_cache_write(p[:, :q_size], p[:, q_size:q_size + kv_size], p[:, q_size + kv_size:q_size + 2 * kv_size] if planes == 2 else None,
                                 positions, token_seq, table, bs, want, inv_freq, rot, neox, nh, nkv, hd, flag)
        cache = torch.zeros_like(want)
        out = torch.full((M, N if extra else q_size), float("nan"), device="cuda", dtype=torch.bfloat16)
        kernels.gemm_skinny_qkv_rope(out, x, w, positions, token_seq, table, bs, cache, inv_freq, rot, neox, nh, nkv, hd, flag, kv_planes=planes,
                                     n_extra=extra, **kw)
        assert flag.item() == 0
        assert torch.equal(out[:, :q_size].view(torch.int16), p[:, :q_size].view(torch.int16))
        assert torch.equal(cache.view(torch.int16), want.view(torch.int16))
        if extra:
            assert torch.equal(out[:, q_size + kv_size:].view(torch.int16), p[:, q_size + kv_size:].view(torch.int16))
