"""The gate and up products with their activation in one tcgen05 kernel (csrc/gemm_gated_tc.cu), against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,I,K", [(1, 8, 8), (17, 128, 64), (128, 136, 72), (129, 120, 200), (256, 1024, 4096), (257, 264, 448),
                                   (600, 1408, 136), (4500, 512, 512), (9000, 384, 64), (2100, 6000, 448), (5000, 2568, 840)])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh"])
def test_gate_and_up_with_their_activation(T, I, K, act):
    """Edges of the tiles of 256 tokens, 128 features and 64 values of k; more than one band of tokens; rows of x and of the output longer
    than what is used; pairs of CTAs that take five tiles and more in turn, whose accumulators and rings are used again and again (the
    ring's six stages run on over the edge between two tiles of 7 and of 14 steps, and are awaited once more at the end).  The result is rounded to
    bfloat16 once (2^-8 of its value) from float32 sums, whose partial results the tensor cores may cut off rather than round (K 2^-23 of the
    sums of the terms' absolute values), passed on by the other factor and by the activation's slope, which is below 1.2."""
    from lmsf_b200 import kernels
    d = torch.device("cuda:0")
    if T * I > 10 ** 7:
        assert -(-T // 256) * -(-I // 128) >= 5 * (kernels.sm_count(d) // 2)
    g = torch.Generator(device=d).manual_seed(T + I + K)
    x = torch.randn((T, K + 8), generator=g, device=d).to(torch.bfloat16)[:, :K]
    w = (torch.randn((2 * I, K), generator=g, device=d) * K ** -0.5).to(torch.bfloat16)
    out = torch.full((T, I + 8), 7.0, dtype=torch.bfloat16, device=d)
    flag = torch.zeros(1, dtype=torch.int32, device=d)
    kernels.gemm_gated_tc(out[:, :I], x, w, act, flag)
    xd, wd = x.double(), w.double()
    gate, up = (xd @ wd.T).split(I, 1)
    a = torch.nn.functional.silu(gate) if act == "silu" else torch.nn.functional.gelu(gate, approximate="tanh")
    ref = a * up
    sums = (xd.abs() @ wd.abs().T).split(I, 1)
    bound = ref.abs() * 2.0 ** -8 + K * 2.0 ** -23 * (sums[0] * up.abs() * 1.2 + sums[1] * a.abs()) + 1e-6
    assert flag.item() == 0
    assert ((out[:, :I].double() - ref).abs() <= bound).all()
    assert (out[:, I:] == 7.0).all()


def test_refusals():
    from lmsf_b200 import kernels
    z = lambda *s: torch.zeros(s, dtype=torch.bfloat16, device="cuda:0")
    for x, w, out in ((z(4, 12), z(32, 12), z(4, 16)), (z(4, 16), z(24, 16), z(4, 12)), (z(4, 16), z(32, 16), z(5, 16)),
                      (z(4, 24)[:, 4:20], z(32, 16), z(4, 16))):
        with pytest.raises(kernels.KernelError):
            kernels.gemm_gated_tc(out, x, w, "silu")


@pytest.mark.parametrize("act", ["silu", "gelu_tanh"])
def test_a_row_on_either_side_of_the_choice(act):
    """The same rows through a feed-forward of 256 rows, whose gate and up stay in float32 up to the activation, and through one of 257, where the
    library rounds both to bfloat16 first.  A row's result moves with the number of rows beside it, by no more than: gate and up rounded
    (2^-8 of each, passed on by the other factor and by the activation's slope, below 1.2), their product rounded on both sides, all of it
    through the down product, and its own rounding on both sides; the down product's float32 sums differ by K 2^-23 of their terms' absolute
    values, those of gate and up (K 64) by 2^-17, which the factor 1.1 covers."""
    from lmsf_b200 import kernels
    from lmsf_b200.parts import linear
    from lmsf_b200.parts.mlp import GatedMLP
    d = torch.device("cuda:0")
    D, inner = 64, kernels.sm_count(d) // 2 * 128
    assert linear.gated_in_one(256, D, inner, d) and not linear.gated_in_one(257, D, inner, d)
    g = torch.Generator(device=d).manual_seed(11)
    w = (torch.randn((2 * inner, D), generator=g, device=d) * D ** -0.5).to(torch.bfloat16)
    down = (torch.randn((D, inner), generator=g, device=d) * inner ** -0.5).to(torch.bfloat16)
    x = torch.randn((257, D), generator=g, device=d).to(torch.bfloat16)
    part = GatedMLP(hidden_size=D, intermediate_size=inner, activation=act)
    part.set_weights({"gate_up": w, "down": down})
    one, apart = part.forward(None, x[:256]).double(), part.forward(None, x)[:256].double()
    xd, u8 = x[:256].double(), 2.0 ** -8
    gate, up = (xd @ w.double().T).split(inner, 1)
    a = torch.nn.functional.silu(gate) if act == "silu" else torch.nn.functional.gelu(gate, approximate="tanh")
    m = (a * up).abs()
    moved = u8 * (1.2 * gate.abs() * up.abs() + m) + 2 * u8 * m
    y = (a * up) @ down.double().T
    bound = 1.1 * (moved @ down.double().abs().T + 2 * u8 * y.abs()) + inner * 2.0 ** -23 * (m @ down.double().abs().T)
    assert not torch.equal(one, apart)
    assert ((one - apart).abs() <= bound).all()
    # and the side that does not round is the nearer one
    assert (one - y).norm() < (apart - y).norm()


def test_under_capture():
    """Decode batches large enough for the kernel are replayed from graphs: what a launch asks of the device is allowed while one is recorded."""
    from lmsf_b200 import kernels
    d = torch.device("cuda:0")
    g = torch.Generator(device=d).manual_seed(2)
    x = torch.randn((260, 192), generator=g, device=d).to(torch.bfloat16)
    w = torch.randn((2 * 640, 192), generator=g, device=d).to(torch.bfloat16)
    out, again = (torch.zeros((260, 640), dtype=torch.bfloat16, device=d) for _ in range(2))
    kernels.gemm_gated_tc(out, x, w, "silu")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        kernels.gemm_gated_tc(again, x, w, "silu")
    assert not again.any()
    for _ in range(2):
        graph.replay()
    assert torch.equal(out, again)
