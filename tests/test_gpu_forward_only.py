"""A forward pass without a backward pass cuts short sequences differently (nothing is kept): same output either way,
on both sides of every tile border up to three tiles."""
import pytest
import torch

from oracle import lasp_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n", [128, 129, 255, 256, 257, 384])
@pytest.mark.parametrize("d,e", [(64, 64), (128, 128), (64, 128)])
def test_forward_without_backward(n, d, e):
    from lasp_b200 import engine, lightning_attn
    b, h = 2, 5
    q, k, v, _ = O.make_inputs(800 + n, b, h, n, d, e)
    s = O.baseline_slopes(h)
    q, k, v = (t.to(torch.bfloat16) for t in (q, k, v))
    with torch.no_grad():
        alone = lightning_attn(q.to(DEV), k.to(DEV), v.to(DEV), s.to(DEV))
    kept = lightning_attn(q.to(DEV).requires_grad_(True), k.to(DEV), v.to(DEV), s.to(DEV)).detach()
    ref = O.dense_closed_form(q.double(), k.double(), v.double(), s)
    ref = ref[0] if isinstance(ref, tuple) else ref
    for t in (alone, kept):
        assert O.max_rel_err(t.double().cpu(), ref) < 2e-2
    assert O.max_rel_err(alone.float(), kept.float()) < 1e-2
    assert engine.read_status() == 0
