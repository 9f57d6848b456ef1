"""The flags by which CTAs of one launch hand states on: stored as a release and read as an acquire, so that the order holds by
the memory model and not by when a fence of another thread happens to be done."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lasp_b200", "csrc")


def test_flags_between_ctas():
    with open(os.path.join(CSRC, "walk_kernels.cu")) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    stores = re.findall(r"(\w+)\((?:a\.sync \+ kSyncFlags \+|ready)(?!.*nothing_published)", code)
    assert stores.count("st_release_u32") == 3 and stores.count("red_release_inc") == 1 and stores.count("wait_flag_eq") == 4, stores
    assert set(stores) == {"st_release_u32", "red_release_inc", "wait_flag_eq"}, stores
    wait = code[code.index("bool wait_flag_eq("):code.index("struct Link")]
    assert "ld_acquire_u32" in wait and "ld_volatile" not in wait
    assert "st.release.gpu" in code and "red.release.gpu" in code and "ld.acquire.gpu" in code
