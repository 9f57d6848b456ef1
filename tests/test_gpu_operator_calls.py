"""The native operator under PyTorch's own machinery: what an autograd function in Python took has to keep working."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _inputs(seed, n=200, dtype=torch.bfloat16):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return [torch.randn(1, 2, n, 64, generator=g, device=DEV).to(dtype) for _ in range(3)]


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("fused", [False, True])
def test_a_traced_function_computes(grad, fused, tmp_path):
    """torch.jit.trace: the graph holds the operator itself, not the allocation of its output alone."""
    from lasp_b200 import lightning_attn, lightning_attn_fused
    s = torch.full((2, 1, 1), 0.01, device=DEV)

    def f(q, k, v):
        return lightning_attn_fused(q, k, v, s, 0.125, "elu1") if fused else lightning_attn(q, k, v, s)

    first = _inputs(1)
    first[0].requires_grad_(grad)
    traced = torch.jit.trace(f, first, check_trace=False)
    path = str(tmp_path / "traced.pt")
    traced.save(path)
    for g in (traced, torch.jit.load(path)):
        q, k, v = _inputs(2)
        q.requires_grad_(grad)
        got, want = g(q, k, v), f(q, k, v)
        assert torch.equal(got, want)
        if grad:
            assert torch.equal(*(torch.autograd.grad(o, q, torch.ones_like(o))[0] for o in (got, want)))


def test_decay_rates_that_require_grad():
    """They are part of the graph (o requires grad on their account alone) and get no gradient."""
    from lasp_b200 import lightning_attn
    q, k, v = _inputs(3)
    s = torch.full((2, 1, 1), 0.01, device=DEV, requires_grad=True)
    o = lightning_attn(q, k, v, s * 1.0)
    assert o.requires_grad
    o.sum().backward()
    assert s.grad is None and q.grad is None
    q.requires_grad_(True)
    with_s = torch.autograd.grad(lightning_attn(q, k, v, s), (q, s), torch.ones_like(o), allow_unused=True)
    without = torch.autograd.grad(lightning_attn(q, k, v, s.detach()), q, torch.ones_like(o))[0]
    assert with_s[1] is None and torch.equal(with_s[0], without)
    with torch.no_grad():
        assert not lightning_attn(q, k, v, s).requires_grad
