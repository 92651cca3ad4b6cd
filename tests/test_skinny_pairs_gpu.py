"""The product of a few rows into the residual, K shared by one block of 16 warps a tile or by a cluster of two blocks."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 5, 8])
@pytest.mark.parametrize("K", [2056, 4096, 4104, 8200])
def test_the_same_bits(cuda_device, M, K):
    """The first columns of a wide product (148 tiles: one block each) and those columns alone (75 tiles: one block, 74 and fewer: two), with a ragged last tile."""
    _same_bits(M, K)


@pytest.mark.parametrize("M", [9, 16])
@pytest.mark.parametrize("K", [2056, 4104])
def test_more_rows_keep_to_one_block(cuda_device, M, K):
    """From nine rows on one block takes a tile however few the tiles are: the same columns, the same bits."""
    _same_bits(M, K)


def _same_bits(M, K):
    from infinilm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + K)
    N = 148 * 16
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) / math.sqrt(K)).bfloat16()
    b, nw, resid = torch.randn(N, device="cuda", generator=g), torch.rand(N, device="cuda", generator=g) + 0.5, torch.randn(M, N, device="cuda", generator=g)

    def run(n, static):
        r, xw, sq = resid[:, :n].clone(memory_format=torch.contiguous_format), torch.empty(M, n, device="cuda", dtype=torch.bfloat16), torch.empty(M, (n + 15) // 16, device="cuda")
        ops.gemm_skinny_resid(x, w[:n], 0.7, b[:n].contiguous(), r, 0.4, nw[:n].contiguous(), 1e-5, xw, sq, w_static=static)
        return r, xw, sq
    r, xw, sq = run(N, True)
    y = 0.7 * (x.double() @ w.double().t()) + b.double()
    assert float((r.double() - (resid.double() + 0.4 * y)).abs().amax()) <= 2.0 ** -8 * 0.4 * float(y.abs().amax())        # the branch is rounded to bfloat16
    for n, static in ((75 * 16, True), (74 * 16, True), (40 * 16, False), (5 * 16 + 3, True), (7, False)):
        r2, xw2, sq2 = run(n, static)
        assert torch.equal(r2, r[:, :n]) and torch.equal(xw2, xw[:, :n]) and torch.equal(sq2[:, :n // 16], sq[:, :n // 16])
