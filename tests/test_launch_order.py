"""Kernels that let the next one start early (programmatic dependent launch): what starts early may rely on everything but the
kernel right before it being complete, so a kernel waits for its own predecessor first; and what the kernel before still
writes is not read-only, so nothing goes by the read-only path."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lasp_b200", "csrc")
SOURCES = ["common.cuh", "split_kernels.cu", "state_kernels.cu"]


def code_of(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_the_wait_comes_before_the_next_kernel_is_let_in():
    for name in SOURCES:
        let_in = r"let_next_start\(\);|griddepcontrol\.launch_dependents"
        for kernel in re.split(r"(?m)^(?=template|__global__|__device__)", code_of(name)):
            opened = re.search(let_in, kernel)
            if opened is None or "void let_next_start()" in kernel:
                continue
            waited = re.search(r"after_previous\(\);|griddepcontrol\.wait", kernel)
            assert waited is not None and waited.start() < opened.start(), f"{name}: {kernel[:120]}"


@pytest.mark.parametrize("name,kernels", [("split_kernels.cu", ["k_split_states", "k_split_out"]), ("state_kernels.cu", ["k_scan"])])
def test_nothing_is_read_by_the_read_only_path(name, kernels):
    code = code_of(name)
    if name == "split_kernels.cu":
        assert "__ldg(" not in code and "__restrict__" not in code
        return
    scan = code[code.index("void __launch_bounds__(256) k_scan"):code.index("k_state_combine")]
    for written_before in ("x_in +", "base +"):
        for use in re.finditer(re.escape(written_before), scan):
            assert scan[:use.start()].rstrip("(").endswith("__ldcg(reinterpret_cast<const float4*>"), scan[use.start() - 60:use.end()]
