"""The aligned cluster barriers need a warp's lanes together: they stand in the helpers of common.cuh alone, each behind a __syncwarp."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "infinilm_b200", "csrc")


def test_every_cluster_barrier_is_behind_a_meeting_of_the_warp():
    found = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh", ".h")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = f.read()
        for m in re.finditer(r'asm volatile\("barrier\.cluster', text):
            assert name == "common.cuh", f"{name}: a cluster barrier of its own"
            assert re.search(r"__syncwarp\(\);\s*$", text[:m.start()]), f"{name}: a cluster barrier without __syncwarp before it"
            found += 1
    assert found == 2                             # arrive, wait
