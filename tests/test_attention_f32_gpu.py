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
