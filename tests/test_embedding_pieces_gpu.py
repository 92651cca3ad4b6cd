"""Embedding rows in 16-byte pieces and element by element: the same bits as the plain lookup."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,H", [(1, 4), (3, 8), (5, 12), (2, 33), (9, 2040), (7, 2052), (64, 2056), (65, 4104), (300, 1024), (1, 10240)])
@pytest.mark.parametrize("shift", [0, 1])
def test_rows(cuda_device, dtype, T, H, shift):
    """shift: the table begins one element past an aligned address (the general kernel takes the call)."""
    from infinilm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(H)
    V = 97
    table = torch.randn(V * H + 8, device="cuda", generator=g).to(dtype)[shift:shift + V * H].view(V, H)
    ids = torch.randint(0, V, (T,), device="cuda", generator=g, dtype=torch.int32)
    out = torch.full((T + 1, H), float("nan"), device="cuda")
    for rounded in (False, True):
        ops.embed(ids, table, 3.7, out[:T], round_bf16=rounded)
        ref = table.float()[ids.long()] * 3.7
        assert torch.equal(out[:T], ref.bfloat16().float() if rounded else ref)
    assert bool(out[T].isnan().all())
