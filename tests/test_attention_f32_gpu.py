"""Float32 attention: the kernel that brings keys and values through shared memory gives the bits of the general kernel, which
takes any alignment, for every mask, head size and length at the edges of its tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("options", [{}, {"window": 40}, {"window": 40, "keep_first": 5}, {"window": 70, "keep_first": 33}, {"chunk": 48},
                                     {"sigmoid": True}, {"softcap": 5.0}, {"kv_planes": 1}])
@pytest.mark.parametrize("hd,bs", [(16, 16), (32, 8), (48, 16), (64, 16), (64, 1)])
def test_staged_kernel_gives_the_bits_of_the_general_one(hd, bs, options):
    from lmsf_b200 import kernels
    heads, kv, planes = 4, 2, options.get("kv_planes", 2)
    g = torch.Generator(device="cuda").manual_seed(hd + bs)
    lens = [1, 2, 31, 32, 33, 127, 128, 129, 300]
    pages = -(-300 // bs)
    n = len(lens) * pages
    size = n * planes * kv * bs * hd
    aligned = torch.randn(size, device="cuda", generator=g).view(n, planes, kv, bs, hd)
    # the same values at an address that is no multiple of 16 bytes: the general kernel
    shifted = torch.empty(size + 1, device="cuda")[1:].view(n, planes, kv, bs, hd).copy_(aligned)
    table = torch.randperm(n, device="cuda", generator=g).to(torch.int32).view(len(lens), pages).contiguous()
    positions = torch.tensor([x - 1 for x in lens], dtype=torch.int32, device="cuda")
    table[-1, 2] = -1                                       # a key without a page is left out
    seq = torch.arange(len(lens), dtype=torch.int32, device="cuda")
    q = torch.randn(len(lens), heads * hd, device="cuda", generator=g)
    outs = []
    for cache in (aligned, shifted):
        out = torch.full_like(q, float("nan"))
        kw = dict(options)
        kernels.attention_generic(out, q, cache, table, bs, seq, positions, hd ** -0.5, kw.pop("window", 0), heads, kv, hd, **kw)
        outs.append(out)
    assert bool(torch.isfinite(outs[0]).all()) and torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("hd", [16, 32, 48, 64])
def test_values_behind_scores_of_minus_infinity(hd):
    """Whole tiles of keys that a bias of minus infinity takes out: their values, infinite ones among them, do not reach the result,
    as in the general kernel."""
    from lmsf_b200 import kernels
    heads, kv, bs, n_keys, seen = 4, 2, 16, 256, 64
    g = torch.Generator(device="cuda").manual_seed(hd)
    pages = n_keys // bs
    aligned = torch.randn(pages * 2 * kv * bs * hd, device="cuda", generator=g).view(pages, 2, kv, bs, hd)
    aligned[:(n_keys - seen) // bs, 1] = float("inf")                    # the values of the keys that are not seen
    shifted = torch.empty(aligned.numel() + 1, device="cuda")[1:].view(aligned.shape).copy_(aligned)
    table = torch.arange(pages, dtype=torch.int32, device="cuda").view(1, pages)
    dist = torch.zeros(heads, seen + 1, device="cuda")
    dist[:, seen] = float("-inf")                                        # 64 keys and more away
    positions, seq = torch.tensor([n_keys - 1], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    q = torch.randn(1, heads * hd, device="cuda", generator=g)
    outs = []
    for cache in (aligned, shifted):
        out = torch.full_like(q, float("nan"))
        kernels.attention_generic(out, q, cache, table, bs, seq, positions, hd ** -0.5, 0, heads, kv, hd, dist=dist)
        outs.append(out)
    assert bool(torch.isfinite(outs[1]).all()) and torch.equal(outs[0], outs[1])


def test_a_bias_per_head_that_the_launch_before_has_written():
    """The bias is read after the launch before it has ended, as q is: made by a product that lets its successor start early, it
    gives the bits of a bias that was there before."""
    from lmsf_b200 import kernels
    heads, kv, hd, bs, pages, K = 16, 8, 64, 16, 4, 65536
    g = torch.Generator(device="cuda").manual_seed(3)
    cache = torch.randn(pages, 2, kv, bs, hd, device="cuda", generator=g)
    table = torch.arange(pages, dtype=torch.int32, device="cuda").view(1, pages)
    positions, seq = torch.tensor([pages * bs - 1], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    q = torch.randn(1, heads * hd, device="cuda", generator=g)
    x, weight = torch.randn(1, K, device="cuda", generator=g) * K ** -0.5, torch.randn(heads, K, device="cuda", generator=g)
    bias = torch.empty(heads, device="cuda")
    out, want = torch.empty_like(q), torch.empty_like(q)

    def make():
        bias.fill_(float("nan"))
        torch.cuda.synchronize()
        kernels.gemm_tn_simt(bias.view(1, heads), x, weight, w_constant=True)

    def attend(to):
        # sigmoid weights: a bias, unlike under a softmax, changes the result
        kernels.attention_generic(to, q, cache, table, bs, seq, positions, hd ** -0.5, 0, heads, kv, hd, sigmoid=True, head_bias=bias)

    make()
    torch.cuda.synchronize()
    attend(want)
    assert bool(torch.isfinite(want).all())
    for _ in range(5):
        make()
        attend(out)
        assert torch.equal(out, want)
