"""What the full-precision kernels compute on the way has 24 bits for 16-bit tensors too: the rank states, which are fp32,
and the results up to the one rounding to their type, against fp64."""
import pytest
import torch

from oracle import lasp_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _all(q, k, v, do, s, dtype):
    from lasp_b200 import engine
    b, h, n, d = q.shape
    e = v.shape[-1]
    plan = engine.make_plan(b, h, n, d, e, dtype, "simt")
    t = [x.to(DEV, dtype) for x in (q, k, v, do)]
    kv, dkv = (torch.empty(b, h, d, e, device=DEV) for _ in range(2))
    fw = engine.Forward(plan, *t[:3], s.to(DEV), kv_out=kv)
    fw.run()
    bw = engine.Backward(plan, *t, s.to(DEV), fw.ws, dkv_out=dkv)
    bw.run()
    torch.cuda.synchronize()
    assert engine.read_status() == 0
    x = [t.to(dtype).double() for t in (q, k, v, do)]
    o, kv_ref = O.blocked_forward(*x[:3], s, dtype=torch.float64)
    *grads, dkv_ref = O.blocked_backward(*x[:3], s, x[3], dtype=torch.float64)
    return (fw.o, bw.dq, bw.dk, bw.dv), (o, *grads), (kv, dkv), (kv_ref, dkv_ref)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d,e,n", [(16, 128, 100), (64, 64, 128), (128, 64, 391), (96, 112, 1000), (128, 128, 2048)])
@pytest.mark.parametrize("slope", [0.0, 0.01, 0.7])
def test_error_against_fp64(dtype, d, e, n, slope):
    s = torch.full((2, 1, 1), slope)
    got, ref, states, state_refs = _all(*O.make_inputs(900 + n, 1, 2, n, d, e), s, dtype)
    # a sum of n products in fp32: n^(1/2) rounding errors of 2^-24 at most, where the largest element is at least as
    # large as the sum of one chunk
    for t, w in zip(states, state_refs):
        assert O.max_rel_err(t, w) < 1e-6
    # one rounding to the type, half a unit in the last place of the element (fp32: the sums' own 24 bits, twice)
    unit = {torch.float32: 0.0, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[dtype]
    for t, w in zip(got, ref):
        err = (t.double().cpu() - w).abs() - unit * w.abs()
        assert (err.max() / w.abs().max()).item() < 2e-6


@pytest.mark.parametrize("small", range(2))
def test_subnormal_fp16_inputs(small):
    """The smallest fp16 numbers, multiples of 2^-24, in q or k."""
    t = list(O.make_inputs(910, 1, 2, 300, 64, 64))
    t[small] *= 2.0 ** -18
    t[2] *= 1e4
    t[3] *= 1e4
    s = torch.full((2, 1, 1), 0.02)
    got, ref, states, state_refs = _all(*t, s, torch.float16)
    for t, w in zip(states, state_refs):
        assert O.max_rel_err(t, w) < 1e-6
    for t, w in ((got[0], ref[0]), (got[3], ref[3])):
        err = (t.double().cpu() - w).abs() - 2.0 ** -11 * w.abs() - 2.0 ** -25
        assert (err.max() / w.abs().max()).item() < 2e-6
