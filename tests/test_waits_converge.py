"""Tensor-memory loads and stores are instructions of a whole warp, undefined where its lanes are apart, and a bounded wait
lets the lanes go one by one: no kernel goes from such a wait to them without bringing the lanes together."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lasp_b200", "csrc")


@pytest.mark.parametrize("name", ["walk_kernels.cu", "wide_kernels.cu", "split_kernels.cu"])
def test_lanes_are_together_after_a_wait(name):
    with open(os.path.join(CSRC, name)) as f:
        lines = f.read().split("\n")
    waits = 0
    for i, line in enumerate(lines):
        if "wait_or_fault(" not in line:
            continue
        for j in range(i + 1, len(lines)):
            text = lines[j].split("//")[0]
            if re.search(r"tc_fence_after_wait|__syncwarp|named_sync|__syncthreads", text):
                waits += 1
                break
            if re.search(r"\btmem_(ld|st)\d|scale_tmem32|stage_row32|masked_pack32|tc_fence_after_sync", text):
                # one thread on its own (an issuer or producer) has no lanes to wait for
                alone = any("lane == 0" in x for x in lines[max(0, i - 12):i])
                assert alone, f"{name}:{i + 1}: {line.strip()} -> {name}:{j + 1}: {lines[j].strip()}"
                break
    assert waits > 0
