"""The 32-bit product in bfloat16 pieces: the error of 32-bit arithmetic, numbers that have no pieces, and every way its sums are cut."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def product(x, w):
    from infinilm_b200 import ops
    out = torch.full((x.shape[0], w.shape[0]), float("nan"), device="cuda")
    ops.gemm_f32(x, w, out)
    ops.check_status(torch.device("cuda:0"))
    return out


@pytest.mark.parametrize("K", [16, 64, 256, 257, 512, 520, 1024, 1056, 2048, 4096])
@pytest.mark.parametrize("spread", [0, 12])
def test_error_of_32_bit_sums(cuda_device, K, spread):
    """Two roundings of 2^-24 a chunk of 64 and one a chunk added, of partial sums that grow with the root of K: below 2^-23 of the result
    together for operands of one size, 1.5 x 2^-23 where a few products decide the sum. (Chains of multiply-adds have 1.1e-7 to 1.5e-7.)"""
    g = torch.Generator(device="cuda").manual_seed(K + spread)
    x, w = (torch.randn(n, K, device="cuda", generator=g) * torch.exp2(torch.randint(-spread, spread + 1, (n, K), device="cuda", generator=g).float())
            for n in (300, 260))
    out, ref = product(x, w), x.double() @ w.double().t()
    assert float((out.double() - ref).norm() / ref.norm()) <= (1.5 if spread else 1.0) * 2.0 ** -23
    for rows in (1, 4, 5, 9, 16, 17, 64, 65):                         # every kernel and cut gives the same bits
        assert torch.equal(product(x[:rows].contiguous(), w), out[:rows]), rows


@pytest.mark.parametrize("M", [3, 16, 40])
def test_numbers_without_pieces(cuda_device, M):
    """Infinities, not-a-numbers, numbers whose rounding overflows and numbers below the range of the lowest piece: what 32-bit
    multiply-adds give, to rounding; the other rows as they are without them."""
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = torch.randn(M, 200, device="cuda", generator=g), torch.randn(150, 200, device="cuda", generator=g)
    clean = product(x, w)
    x[0, 3] = float("inf")
    x[1, 5], x[1, 6] = float("nan"), 1.0
    x[2] *= 2.0 ** -125
    w[7, 3], w[8] = 0.0, 0.0
    w[9] *= 2.0 ** -120
    out, ref = product(x, w), x.double() @ w.double().t()
    assert torch.equal(out[0].isnan(), ref[0].isnan()) and torch.equal(out[0].isinf(), ref[0].isinf()) and bool(out[1].isnan().all())
    live = torch.ones(150, dtype=torch.bool, device="cuda")
    live[7], live[8], live[9] = False, False, False
    size = x[2].double().abs() @ w.double().abs().t()
    assert bool(((out[2].double() - ref[2]).abs() <= 204 * (2.0 ** -24 * size + 2.0 ** -149)).all())      # (a rounding a product, or the smallest number)
    assert bool((out[3:, 8] == 0).all()) and torch.equal(out[3:][:, live], clean[3:][:, live])
    # (signs change every second place: even and odd places are summed apart, and 32 of one sign would overflow in any order)
    big = torch.full((M, 64), 3.4e38, device="cuda") * torch.where(torch.arange(64, device="cuda") % 4 < 2, 1.0, -1.0)
    assert bool(product(big, torch.full((20, 64), 2.0 ** -3, device="cuda")).abs().max() <= 3.4e38 * 2.0 ** -20)
    assert bool(product(x[2:], torch.zeros(20, 200, device="cuda")).eq(0).all())
