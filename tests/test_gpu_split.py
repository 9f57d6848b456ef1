"""The full-precision tensor-core kernels (fp32 and fp16, and bf16 shapes outside the walk kernels) at the edges of
their 128-token chunks and 64/128-wide operand tiles, against the fp64 closed form."""
import pytest
import torch

from oracle import lasp_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype,gate", [(torch.float32, 3e-6), (torch.float16, 2e-3), (torch.bfloat16, 1e-2)])
@pytest.mark.parametrize("shape", [(1, 2, 1, 16, 16), (1, 2, 127, 64, 80), (2, 1, 128, 80, 64), (1, 3, 129, 16, 128),
                                   (1, 2, 257, 112, 16), (1, 80, 260, 128, 48), (1, 2, 140, 272, 144)])
@pytest.mark.parametrize("slope", [0.0, 0.05, 2.0])
def test_full_precision_kernels_at_tile_edges(dtype, gate, shape, slope):
    from lasp_b200 import engine, lightning_attn
    b, h, n, d, e = shape
    q, k, v, do = (t.to(dtype) for t in O.make_inputs(700 + n + d, b, h, n, d, e))
    s = torch.full((h, 1, 1), slope)
    dev = [t.to(DEV).requires_grad_(i < 3) for i, t in enumerate((q, k, v, do))]
    o = lightning_attn(*dev[:3], s.to(DEV))
    got = (o, *torch.autograd.grad(o, dev[:3], dev[3]))
    ref = O.dense_closed_form(*(t.double() for t in (q, k, v)), s, do.double())
    for t, w, key in zip(got, ref, ("o", "dq", "dk", "dv")):
        assert O.max_rel_err(t.detach().double().cpu(), w) < gate, key
    assert engine.read_status() == 0
