"""The 32-bit product where an operand's bfloat16 pieces leave their range: the error of 32-bit multiply-adds all the same, and nothing of it in the rows beside."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def product(x, w):
    from infinilm_b200 import ops
    out = torch.full((x.shape[0], w.shape[0]), float("nan"), device="cuda")
    ops.gemm_f32(x, w, out)
    ops.check_status(torch.device("cuda:0"))
    return out


def close(out, x, w):
    """Sums of 32 products in a row, two of these, the small products and K / 64 chunks: a rounding of 2^-24 of at most the sum of the sizes each; a product
    below the normal range is rounded to a multiple of 2^-149."""
    K = x.shape[1]
    x, w = x.double(), w.double()
    bound = (36 + (K + 63) // 64) * 2.0 ** -24 * (x.abs() @ w.abs().t()) + K * 2.0 ** -149
    return bool(((out.double() - x @ w.t()).abs() <= bound).all())


# a few rows in shared memory and not, K in one block and over a cluster; clusters of tiles, blocks of their own
SHAPES = [(1, 150, 256), (3, 150, 1056), (8, 150, 257), (16, 150, 1024), (40, 150, 1024), (300, 2100, 320)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("tiny,large", [(-104, 30), (-110, 40), (-120, 60), (-126, 120), (-118, 118), (-136, 100), (-141, 110), (-141, 0), (-70, -75), (-130, -10)])
def test_small_operands_against_large(cuda_device, M, N, K, tiny, large):
    g = torch.Generator(device="cuda").manual_seed(M + K - tiny)
    x, w = torch.randn(M, K, device="cuda", generator=g), torch.randn(N, K, device="cuda", generator=g) * 2.0 ** large
    x[:, ::7] = 0.0
    w[11] = 0.0
    clean = product(x, w)
    assert close(clean, x, w)
    x[0] *= 2.0 ** tiny                           # a row of activations ...
    one = x.clone()
    if M > 1:
        one[1, 3::5] *= 2.0 ** tiny               # ... some numbers of another ...
    out = product(one, w)
    assert close(out, one, w)
    assert torch.equal(out[2:], clean[2:]) and bool(out[:, 11].eq(0).all())
    v = torch.randn(N, K, device="cuda", generator=g)
    v[7] *= 2.0 ** tiny                           # ... or a row of weights
    big = torch.randn(M, K, device="cuda", generator=g) * 2.0 ** large
    whole = product(big, v)
    assert close(whole, big, v)
    v[7] = 1.0
    same = product(big, v)
    live = torch.arange(N, device="cuda") != 7
    assert torch.equal(whole[:, live], same[:, live])


@pytest.mark.parametrize("M,K", [(1, 1024), (4, 300), (7, 2048), (16, 1024)])
@pytest.mark.parametrize("tiny,large", [(-120, 119), (-134, 124)])
def test_gated_product(cuda_device, M, K, tiny, large):
    from infinilm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + K)
    x, w = torch.randn(M, K, device="cuda", generator=g) * 2.0 ** tiny, torch.randn(180, K, device="cuda", generator=g) * 2.0 ** large * K ** -0.5
    out = torch.empty(M, 90, device="cuda")
    ops.gemm_f32(x, w, out, glu=ops.ACT_SILU)
    y = x.double() @ w.double().t()
    ref = torch.nn.functional.silu(y[:, :90]) * y[:, 90:]
    # two sums of a few units with an error of some 2^-22 each, and a short function
    assert float((out.double() - ref).abs().max()) <= 2.0 ** -18 * float(ref.abs().max())


def test_one_small_number_among_large_ones(cuda_device):
    """The rows beside it keep their bits, and the row has the same bits alone."""
    g = torch.Generator(device="cuda").manual_seed(9)
    x, w = torch.randn(33, 1024, device="cuda", generator=g) * 2.0 ** 40, torch.randn(200, 1024, device="cuda", generator=g) * 2.0 ** 60
    clean = product(x, w)
    x[5, 100] = 2.0 ** -125
    out = product(x, w)
    rest = torch.arange(33, device="cuda") != 5
    assert torch.equal(out[rest], clean[rest]) and torch.equal(product(x[5:6].contiguous(), w), out[5:6]) and close(out, x, w)
