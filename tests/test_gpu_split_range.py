"""The full-precision kernels outside the range of their bf16 terms: infinities, NaN and fp32 values above bf16's largest
(3.39e38) come out, and reach as far, as plain fp32 arithmetic lets them."""
import pytest
import torch

from oracle import lasp_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
INF = float("inf")


def _run(q, k, v, do, s, dtype):
    from lasp_b200 import engine, lightning_attn
    t = [x.to(DEV, dtype).requires_grad_(i < 3) for i, x in enumerate((q, k, v, do))]
    o = lightning_attn(*t[:3], s.to(DEV))
    out = [x.detach().float().cpu() for x in (o, *torch.autograd.grad(o, t[:3], t[3]))]
    assert engine.read_status() == 0
    return out


@pytest.mark.parametrize("dtype,width", [(torch.float32, 48), (torch.float16, 48), (torch.bfloat16, 48),
                                         (torch.float32, 144), (torch.float16, 144)])   # 144: slices that are added up
@pytest.mark.parametrize("token", [0, 100, 127, 128, 299])
@pytest.mark.parametrize("value", [INF, -INF, float("nan")])
def test_what_is_not_finite_reaches_the_tokens_it_reaches(dtype, width, token, value):
    """One such value in k, or in v, at one token of 300 (three chunks): the results of the tokens before it are as without
    it, those from it on have the infinity's sign or are NaN - and the mirror image in the gradients.  (Beyond the token's
    chunk of 128 a state of infinities of both signs gives NaN where the dense form gives an infinity.)"""
    n, d = 300, width
    q, k, v, do = (t.to(dtype).float() for t in O.make_inputs(60, 1, 1, n, d, d))
    s = torch.full((1, 1, 1), 0.01)
    plain = _run(q, k, v, do, s, dtype)
    col = 5
    # results next to one that is not finite are summed again in another order: to 24 bits before the rounding to the type
    near = {torch.float32: 1e-5, torch.float16: 2.0 ** -10, torch.bfloat16: 2.0 ** -7}[dtype]
    def times(a, b):                                       # (a sum over the 128-wide slices of q and k)
        return sum(value * (a[:, i:i + 128] @ b[i:i + 128]) for i in range(0, d, 128))

    for name in ("k", "v", "do"):
        t = dict(k=k.clone(), v=v.clone(), do=do.clone())
        t[name][0, 0, token, col] = value
        o, dq, dk, dv = _run(q, t["k"], t["v"], t["do"], s, dtype)
        if name == "k":      # o_r += (q_r,col k_col) v_token for r >= token
            assert torch.equal(o[:, :, :token], plain[0][:, :, :token])
            want = value * q[0, 0, token:, col, None] * v[0, 0, token]
            got = o[0, 0, token:]
        elif name == "v":    # o_r,col += (q_r k_token) v_col
            keep = [c for c in range(d) if c != col]
            assert O.max_rel_err(o[..., keep], plain[0][..., keep]) < near
            assert token == 0 or O.max_rel_err(o[:, :, :token], plain[0][:, :, :token]) < near
            end = min(n, token // 128 * 128 + 128)
            want = times(q[0, 0, token:end].double(), k[0, 0, token].double())
            got = o[0, 0, token:end, col].double()
            assert not torch.isfinite(o[0, 0, end:, col]).any()
        else:                # dv_c,col += (q_token k_c) do_col for c <= token
            for x, y in ((dv, plain[3]), (dk, plain[2])):
                assert token == n - 1 or O.max_rel_err(x[:, :, token + 1:], y[:, :, token + 1:]) < near
            start = token // 128 * 128
            want = times(k[0, 0, start:token + 1].double(), q[0, 0, token].double())
            got = dv[0, 0, start:token + 1, col].double()
            assert not torch.isfinite(dv[0, 0, :start, col]).any()
        assert bool((torch.isnan(want) & torch.isnan(got) | (want == got)).all()), name


def test_values_above_the_largest_bf16():
    """fp32 inputs of 3.4e38 with results that fp32 holds, against fp64."""
    n, d = 260, 64
    q, k, v, do = O.make_inputs(61, 1, 2, n, d, d)
    s = torch.tensor([0.0, 0.05]).reshape(2, 1, 1)
    for big in range(4):
        t = [x * 1e-12 for x in (q, k, v, do)]             # (the results stay inside fp32)
        t[big] *= 1e12
        t[big][0, :, 40, 3], t[big][0, :, 200, 7] = 3.4e38, -3.395e38
        got = _run(*t, s, torch.float32)
        ref = O.dense_closed_form(*(x.double() for x in t[:3]), s, t[3].double())
        for x, w, key in zip(got, ref, ("o", "dq", "dk", "dv")):
            assert bool(torch.isfinite(w.float()).all()), (big, key)
            assert O.max_rel_err(x, w) < 3e-6, (big, key)
