"""256-wide heads in bf16, each result in one pass (csrc/wide_kernels.cu), on both sides of the rule that chooses between it
and the 128-wide slices."""
import ctypes as C

import pytest
import torch

from oracle import lasp_oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("decay", [False, True])
@pytest.mark.parametrize("shape", [(1, 1, 128), (1, 2, 129), (2, 1, 255), (1, 3, 384), (5, 31, 200), (1, 2, 1500), (1, 2, 6001)])
def test_wide_heads_against_the_blocked_recurrence(shape, decay):
    """One tile, a tile and a token, a last tile of 127, more items than SMs; at 1500 tokens the forward pass goes by slices and
    the backward pass does not, at 6001 both go by slices."""
    from lasp_b200 import engine, lightning_attn
    b, h, n = shape
    q, k, v, do = (t.to(torch.bfloat16) for t in O.make_inputs(n + h, b, h, n, 256, 256))
    s = O.baseline_slopes(h) if decay else torch.zeros(h, 1, 1)
    dev = [t.to("cuda:0").requires_grad_(i < 3) for i, t in enumerate((q, k, v, do))]
    o = lightning_attn(*dev[:3], s.to("cuda:0"))
    got = (o, *torch.autograd.grad(o, dev[:3], dev[3]))
    with torch.no_grad():
        alone = lightning_attn(*dev[:3], s.to("cuda:0"))
    heads = slice(0, h) if b * h <= 6 else slice(h - 2, h)     # (the oracle on a few heads of a large call)
    x = [t[-1:, heads].float() for t in (q, k, v, do)]
    ref = O.fwd_bwd(*x[:3], s[heads], x[3])
    assert O.max_rel_err(alone[-1:, heads].float().cpu(), ref[0]) < 2e-2
    for t, w, key in zip(got, ref, ("o", "dq", "dk", "dv")):
        assert O.max_rel_err(t[-1:, heads].detach().float().cpu(), w) < 2e-2, key
    assert engine.read_status() == 0


def test_what_is_refused():
    """The entry points check before anything is launched (no GPU needed)."""
    from lasp_b200 import _cabi
    lib = _cabi.load()

    def problem(**kw):
        return C.byref(_cabi.Problem(**{**dict(b=4, h=16, n=4096, d=256, e=256, dtype=_cabi.BF16), **kw}))

    assert lib.lasp_b200_wide_ok(problem(), 0) == 1 and lib.lasp_b200_wide_ok(problem(), 1) == 1
    assert lib.lasp_b200_wide_ok(problem(b=1, h=2, n=65536), 0) == 0 and lib.lasp_b200_wide_ok(problem(b=1, h=2, n=65536), 1) == 0
    for kw, status in (dict(d=128), -2), (dict(e=192), -2), (dict(n=127), -2), (dict(pitch_d=512), -2), (dict(dtype=_cabi.F32), -7), \
            (dict(dtype=9), -3), (dict(qk_map=1), -7), (dict(qk_scale=0.5), -7), (dict(path=_cabi.PATH_SIMT), -7), (dict(h=20000), -2):
        assert lib.lasp_b200_wide_ok(problem(**kw), 0) == status, kw
    p = problem()
    fwd = dict(q=4096, k=4096, v=4096, s=4096, o=4096)
    assert lib.lasp_b200_forward_wide(p, C.byref(_cabi.FwdArgs(**{**fwd, "o": 0})), None) == -1
    assert lib.lasp_b200_forward_wide(p, C.byref(_cabi.FwdArgs(**{**fwd, "q": 4104})), None) == -4
    assert lib.lasp_b200_forward_wide(p, C.byref(_cabi.FwdArgs(**fwd, kv_out=4096)), None) == -2
    bwd = dict(q=4096, k=4096, v=4096, d_o=4096, s=4096, dq=4096, dk=4096, dv=4096)
    assert lib.lasp_b200_backward_wide(p, C.byref(_cabi.BwdArgs(**{**bwd, "dk": 0})), None) == -1
    assert lib.lasp_b200_backward_wide(p, C.byref(_cabi.BwdArgs(**{**bwd, "dv": 4104})), None) == -4
    assert lib.lasp_b200_backward_wide(p, C.byref(_cabi.BwdArgs(**bwd, dkv_in=4096)), None) == -2
