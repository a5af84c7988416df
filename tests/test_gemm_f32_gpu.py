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


@pytest.mark.parametrize("M", [1, 3, 16])
def test_a_second_operand_that_the_launch_before_has_written(M):
    """Only what the caller calls a weight is read ahead of the launch before: a product whose w is the output of a product that lets
    its successor start early gives the bits that it gives when everything before it has ended."""
    from lmsf_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(M)
    rows, K, N = 16, 4096, 8192                              # the first product takes tens of microseconds
    x, weight = torch.randn(rows, K, device="cuda", generator=g), torch.randn(N, K, device="cuda", generator=g)
    a = torch.randn(M, N, device="cuda", generator=g)
    w = torch.empty(rows, N, device="cuda")
    out, want = torch.empty(M, rows, device="cuda"), torch.empty(M, rows, device="cuda")
    w3, a3 = w.view(4, 4, N), a.view(M, 4, N // 4)           # as a batch: w[b] = rows 4 b .. of w, its first N / 4 values
    out3, want3 = torch.empty(M, 4, 4, device="cuda"), torch.empty(M, 4, 4, device="cuda")

    def first():
        w.fill_(float("nan"))
        torch.cuda.synchronize()
        kernels.gemm_tn_simt(w, x, weight, w_constant=True)

    first()
    torch.cuda.synchronize()
    kernels.gemm_tn_simt(want, a, w)
    kernels.gemm_tn_simt_batched(want3, a3, w3[:, :, :N // 4])
    assert bool(torch.isfinite(want).all()) and bool(torch.isfinite(want3).all())
    for _ in range(5):
        first()
        kernels.gemm_tn_simt(out, a, w)
        assert torch.equal(out, want)
        first()
        kernels.gemm_tn_simt_batched(out3, a3, w3[:, :, :N // 4])
        assert torch.equal(out3, want3)
    # the second one as what it is, after a synchronisation: the same bits
    kernels.gemm_tn_simt(out, a, w, w_constant=True)
    assert torch.equal(out, want)
