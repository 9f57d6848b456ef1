"""Span totals over more tiles than the ring that streams them has stages, at every mix of head widths: slowly decaying
heads (the total takes all tiles), fast ones (the sums stop early) and a ragged tail."""
import pytest
import torch

from oracle import lasp_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("d,e", [(128, 128), (128, 64), (64, 128), (64, 64)])
@pytest.mark.parametrize("n", [8 * 128, 21 * 128 - 37])
def test_totals_longer_than_the_ring(d, e, n):
    from lasp_b200 import engine, lightning_attn
    h, heads = 72, [0, 35, 71]                      # two spans per sequence on 148 SMs
    g = torch.Generator(device=DEV).manual_seed(n + d)
    q, k = (torch.randn(1, h, n, d, device=DEV, generator=g) * d ** -0.5 for _ in range(2))
    v, do = (torch.randn(1, h, n, e, device=DEV, generator=g) for _ in range(2))
    s = torch.zeros(h, 1, 1)
    s[heads[1]], s[heads[2]] = 0.004, 0.2
    q, k, v, do = (t.to(torch.bfloat16) for t in (q, k, v, do))
    for t in (q, k, v):
        t.requires_grad_(True)
    o = lightning_attn(q, k, v, s.to(DEV))
    got = (o, *torch.autograd.grad(o, (q, k, v), do))
    ref = O.fwd_bwd(*(t.detach()[:, heads].float().cpu() for t in (q, k, v)), s[heads], do[:, heads].float().cpu())
    for t, w, key in zip(got, ref, ("o", "dq", "dk", "dv")):
        for i, head in enumerate(heads):
            assert O.max_rel_err(t.detach()[:, head].float().cpu(), w[:, i]) < 2e-2, (key, head)
    assert engine.read_status() == 0
