"""lasp_b200_forward_static over problems of both kernel paths in turn: the full-precision path keeps nothing where the
tensor path keeps the words that its CTAs synchronise through, so a call's CTAs wait for this call's span totals."""
import pytest
import torch

from lasp_b200 import engine
from oracle import lasp_oracle as O
from tests.test_zz_no_alloc import _forward_static

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("before", [torch.float32, torch.float16])
def test_calls_of_both_paths_share_the_scratch(before):
    h, n, d = 72, 2048, 128                            # two spans per sequence: the second sums nothing and only waits
    s = torch.zeros(h, device=DEV)                     # every span's total reaches every later span
    plan = engine.make_plan(1, h, n, d, d, torch.bfloat16)
    first = engine.make_plan(1, h, 512, 64, 64, before)
    q, k, v, _ = O.make_inputs(7, 1, h, 512, 64, 64)
    _forward_static(first, *(t.to(DEV, before) for t in (q, k, v)), s,
                    torch.randn(1, h, 64, 64, device=DEV), None)
    g = torch.Generator(device=DEV).manual_seed(7)
    calls = []
    for _ in range(6):
        q, k, v = ((torch.rand(1, h, n, d, generator=g, device=DEV) + 0.5).to(torch.bfloat16) for _ in range(3))
        calls.append((q, k, v, engine.Forward(plan, q, k, v, s).run()))
    got = [_forward_static(plan, q, k, v, s, None, None) for q, k, v, _ in calls]   # back to back
    for o, (_, _, _, want) in zip(got, calls):
        assert torch.equal(o, want)
    assert engine.read_status() == 0
