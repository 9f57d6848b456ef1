"""What the entry points that take mapped q and k refuse, before anything is launched (no GPU needed)."""
import ctypes as C

import pytest

from lasp_b200 import _cabi


@pytest.fixture(scope="module")
def lib():
    return _cabi.load()


def test_map_qk_arguments(lib):
    good = [4096, 8192, 12288, 16384]
    for i in range(4):
        assert lib.lasp_b200_map_qk(*(None if j == i else p for j, p in enumerate(good)), 64, None) == -1
        assert lib.lasp_b200_map_qk(*(p + 8 if j == i else p for j, p in enumerate(good)), 64, None) == -4
    for elements in (0, -8, 4, 12):
        assert lib.lasp_b200_map_qk(*good, elements, None) == -2


def test_who_takes_mapped_input(lib):
    def problem(**kw):
        return C.byref(_cabi.Problem(**{**dict(b=2, h=12, n=2048, d=128, e=128, dtype=_cabi.BF16), **kw}))

    assert lib.lasp_b200_resolve_path(problem(qk_map=2)) == _cabi.PATH_TENSOR
    assert lib.lasp_b200_linked_ok(problem(qk_map=1)) == 1 and lib.lasp_b200_linked_ok(problem(qk_map=2)) == 0
    for kw, status in (dict(qk_map=3), -2), (dict(qk_map=-1), -2), (dict(qk_map=2, dtype=_cabi.F32), -7), (dict(qk_map=2, n=100), -7), \
            (dict(qk_map=2, path=_cabi.PATH_SIMT), -7):
        assert lib.lasp_b200_resolve_path(problem(**kw)) == status, kw
    args = _cabi.FwdArgs(q=4096, k=4096, v=4096, s=4096, o=4096, ws=4096, ws_bytes=1 << 40)
    for phase in ("fwd_chunk_states", "fwd_scan", "fwd_output"):
        assert getattr(lib, f"lasp_b200_{phase}")(problem(qk_map=2), C.byref(args), None) == -7, phase
