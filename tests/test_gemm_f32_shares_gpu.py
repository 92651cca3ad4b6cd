"""The 32-bit product where K is cut over the two blocks of a cluster, and where it is not: the same bits for a row whatever the shape."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [64, 511, 1024, 1030, 2047, 2050, 4096, 4100, 14336])
@pytest.mark.parametrize("M,N", [(17, 40), (61, 1024), (150, 200), (300, 1000), (800, 1024), (513, 2049)])
def test_shares(cuda_device, M, N, K):
    from infinilm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + K)
    x = torch.randn(M, K, device="cuda", generator=g)
    w = torch.randn(N, K, device="cuda", generator=g) / math.sqrt(K)
    b = torch.randn(N, device="cuda", generator=g) if M % 2 else None
    out = torch.full((M, N + 1), float("nan"), device="cuda")
    ops.gemm_f32(x, w, out[:, :N], 0.5, b)
    ref = 0.5 * (x.double() @ w.double().t()) + (b.double() if b is not None else 0.0)
    # chains of 32 products, of up to K / 64 chunks, a sum of two, and the scale and bias: each at most one rounding of the sum of the magnitudes
    size = 0.5 * (x.abs().double() @ w.abs().double().t()) + (b.abs().double() if b is not None else 0.0)
    assert bool(((out[:, :N].double() - ref).abs() <= (36 + math.ceil(K / 64)) * 2.0 ** -24 * size).all())
    assert bool(out[:, N:].isnan().all())
    few = torch.empty(9, N, device="cuda")
    ops.gemm_f32(x[5:14].contiguous(), w, few, 0.5, b)
    assert torch.equal(few, out[5:14, :N])


def test_millions_of_rows(cuda_device):
    """More rows than 65,535 tiles of 32 or 64 have: the taller tiles take them."""
    from infinilm_b200 import ops
    M, N, K = 4_300_000, 32, 4
    g = torch.Generator(device="cuda").manual_seed(1)
    x, w = torch.randn(M, K, device="cuda", generator=g), torch.randn(N, K, device="cuda", generator=g)
    out = torch.full((M, N), float("nan"), device="cuda")
    ops.gemm_f32(x, w, out)
    for at in (0, 4_194_240 - 8, M - 20):
        few = torch.empty(16, N, device="cuda")
        ops.gemm_f32(x[at:at + 16], w, few)
        assert torch.equal(out[at:at + 16], few)
    assert not bool(out.isnan().any())
