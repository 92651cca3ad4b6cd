"""Every code that a kernel leaves when a bounded wait runs out is reported under that kernel's name."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "infinilm_b200", "csrc")


def test_codes_of_the_sources_are_the_codes_of_the_message():
    from infinilm_b200 import ops
    seen = set()
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name), encoding="utf-8") as fh:
                for code in re.findall(r"atomicExch\((?:\w+\.)?status, (\d+)\)", fh.read()):
                    owner = [n for lo, hi, n in ops.STATUS_CODES if lo <= int(code) <= hi]
                    assert owner == [os.path.splitext(name)[0]], (name, code, owner)
                    seen.add(owner[0])
    assert seen == {n for _, _, n in ops.STATUS_CODES}


def test_the_error_names_the_kernel(monkeypatch):
    import pytest
    import torch

    from infinilm_b200 import ops
    for code, name in ((72, "gemm_f32"), (83, "gemm_narrow_tc5"), (21, "attn_decode"), (99, "no kernel known")):
        word = torch.tensor([code], dtype=torch.int32)
        monkeypatch.setitem(ops._stream_status, 0, word)
        with pytest.raises(ops.KernelError, match=f"code {code}: {name}"):
            ops.check_status("cuda:0")
        assert int(word) == 0                     # asked once, it is cleared
