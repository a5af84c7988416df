"""The float32 product: every kernel of it (few rows, tiles alone, tiles shared by a cluster, any alignment) adds in one
fixed order, so that a row has the same bits whichever of them made it, and its error is that of chains of K / 8 sums."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _product(a, w):
    from lmsf_b200 import kernels
    out = torch.full((a.shape[0], w.shape[0]), float("nan"), device="cuda")
    kernels.gemm_tn_simt(out, a, w)
    return out


@pytest.mark.parametrize("N,K", [(1, 4), (15, 32), (129, 36), (300, 260), (128, 1024), (2048, 516), (257, 2052), (64, 4096), (33, 4612), (40000, 64)])
def test_every_route_gives_the_same_bits(N, K):
    g = torch.Generator(device="cuda").manual_seed(N + K)
    a = torch.randn(700, K, device="cuda", generator=g)
    w = torch.randn(N, K, device="cuda", generator=g)
    exact = a.double() @ w.double().T
    # a chain of n FMAs errs by at most n 2^-24 times the sum of the products' sizes; here no sum has passed through more than
    # K / 16 + 16 FMAs of a chain, its other half and eight parts, and K / 8 + 40 is more
    bound = (math.ceil(K / 8) + 32 + 8) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    whole = _product(a, w)
    assert bool(((whole.double() - exact).abs() <= bound).all())
    for m in (1, 2, 3, 4, 5, 6, 7, 8, 9, 16, 17, 64, 65, 128, 129, 500):
        assert torch.equal(_product(a[-m:], w), whole[-m:]), m
    # rows that cannot be read 16 bytes at a time
    odd_w = torch.empty(N, K + 1, device="cuda")[:, :K].copy_(w)
    assert torch.equal(_product(a[:70], odd_w), whole[:70])
    odd_a = torch.empty(70 * K + 1, device="cuda")[1:].view(70, K).copy_(a[:70])
    assert torch.equal(_product(odd_a, w), whole[:70])


@pytest.mark.parametrize("M,N,K", [(3, 48, 64), (70, 130, 64), (33, 64, 100)])
def test_batches_of_products(M, N, K):
    from lmsf_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(5)
    a = torch.randn(M, 5, K, device="cuda", generator=g)
    w = torch.randn(5, N, K, device="cuda", generator=g)
    out = torch.full((M, 5, N), float("nan"), device="cuda")
    kernels.gemm_tn_simt_batched(out, a, w)
    for b in range(5):
        assert torch.equal(out[:, b], _product(a[:, b].contiguous(), w[b]))
