"""Kernels that may become resident while the kernel in front still runs: what that kernel writes is never read through a
`const __restrict__` pointer, whose loads the compiler may move above the wait (checked in the sources, no GPU)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "infinilm_b200", "csrc")
# Parameters that no kernel of a step writes: weights and tables of the model (and of a request's sampling), and the step's descriptors,
# which the host copies to the device.
WRITTEN_LONG_BEFORE = {
    "W", "w", "bias", "norm_w", "w_a", "w_b", "wq", "wk", "wb", "wn", "corr", "sink", "dist_bias", "table", "pair_table", "inv_freq", "freq", "decay",
    "A_log", "dt_bias", "mix", "out_w", "in_next", "vec",
    "temperature", "top_k", "top_p", "uniform",
    "tok_pos", "tok_entry", "block_table", "entry_qstart", "entry_kvlen", "qstart", "read_slots", "write_slots", "rows", "src_idx",
}
WAIT = re.compile(r"il_pdl_wait|il_pdl_begin|sm_small_begin|gs_begin|griddepcontrol\.wait")
KERNEL = re.compile(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(([^{]*?)\)\s*\{", re.S)
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _waiting_kernels(name):
    with open(os.path.join(CSRC, name), encoding="utf-8") as fh:
        text = re.sub(r"//[^\n]*", "", fh.read())
    for m in KERNEL.finditer(text):
        at, depth = m.end(), 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        if WAIT.search(text[m.end():at]):
            yield m.group(1), m.group(2)


@pytest.mark.parametrize("name", FILES)
def test_what_the_kernel_in_front_writes_is_not_read_only(name):
    bad = []
    for kernel, params in _waiting_kernels(name):
        for p in params.split(","):
            if "__restrict__" in p and re.search(r"\bconst\b", p):
                arg = re.search(r"(\w+)\s*$", p).group(1)
                if arg not in WRITTEN_LONG_BEFORE:
                    bad.append(f"{kernel}: {arg}")
    assert not bad, bad


def test_the_kernels_are_found():
    assert sum(1 for name in FILES for _ in _waiting_kernels(name)) >= 50


@pytest.mark.parametrize("op", ["gemm_f32", "gemm_skinny", "gemm_skinny_resid", "gemm_skinny_rope", "gemm_skinny_gelu_row", "latent_norm_store",
                                "short_conv", "matrix_state_scan"])
def test_reading_before_the_wait_is_for_the_caller_to_allow(op):
    """Kernels that read weights before their wait overlap with the kernel in front only where the caller says that it wrote none of them."""
    import inspect

    from infinilm_b200 import ops
    assert inspect.signature(getattr(ops, op)).parameters["w_static"].default is False


def test_the_experts_gate_product_lets_its_successor_in_behind_its_wait():
    """The experts' back product reads the groups' ranges before its wait: right only while the gate product in front of it, which waits with
    il_pdl_begin, lets nobody in before that. No switch may change it."""
    with open(os.path.join(CSRC, "common.cuh"), encoding="utf-8") as fh:
        common = re.sub(r"//[^\n]*", "", fh.read())
    with open(os.path.join(CSRC, "gemm_grouped.cu"), encoding="utf-8") as fh:
        grouped = re.sub(r"//[^\n]*", "", fh.read())
    body = re.search(r"void il_pdl_begin\(\)\s*\{([^}]*)\}", common).group(1)
    assert body.split() == ["il_pdl_wait();"]
    assert "il_pdl_launch_dependents" not in grouped and "griddepcontrol" not in grouped
    for kernel in re.split(r"__global__", grouped)[1:]:
        wait, tail = re.search(r"il_pdl_(?:wait|begin)\(", kernel), re.search(r"il_pdl_tail\(", kernel)
        assert wait and (tail is None or wait.start() < tail.start())
