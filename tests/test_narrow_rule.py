"""Which rows a narrow model's gated feed-forward gives to the fused decode products (no GPU)."""
import pytest
import torch

from infinilm_b200.parts.feed_forward import SwiGLU


@pytest.mark.parametrize("hidden,inter,rows,fused", [
    (1024, 4096, 48, True), (1024, 4736, 33, True), (1024, 4737, 33, False), (1024, 8192, 48, False), (896, 4864, 33, False),
    (1024, 8192, 32, True), (1024, 8192, 17, True), (1024, 8192, 16, True), (512, 4736, 48, True), (504, 2048, 17, False), (1032, 2048, 17, False), (1024, 2048, 49, False)])
def test_more_blocks_than_sms_end_at_32_rows(hidden, inter, rows, fused):
    ffn = SwiGLU({"hidden": hidden, "intermediate": inter}, "", torch.bfloat16)
    assert ffn.accepts_normed(rows) == fused
    assert not ffn.fuses_tail(rows) or fused
