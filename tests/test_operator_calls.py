"""How the native operator takes calls that are not ordinary ones, as far as it looks at them before it needs a GPU."""
import pytest
import torch


@pytest.mark.parametrize("d,e", [(0, 64), (64, 0), (0, 0)])
@pytest.mark.parametrize("grad", [False, True])
def test_empty_heads_are_refused(d, e, grad):
    """A head width of zero leaves no slice to run: the output must not come back as it was allocated."""
    from lasp_b200 import lightning_attn
    from lasp_b200.engine import LaspStatusError
    q, v = torch.zeros(1, 2, 200, d, requires_grad=grad), torch.zeros(1, 2, 200, e)
    with pytest.raises(LaspStatusError, match="unsupported shape"):
        lightning_attn(q, q, v, torch.zeros(2, 1, 1))


@pytest.mark.parametrize("which", range(4))
@pytest.mark.parametrize("grad", [False, True])
def test_a_tangent_is_refused(which, grad):
    """There is no forward-mode derivative: a dual tensor must not lose its tangent on the way."""
    import torch.autograd.forward_ad as fa
    from lasp_b200 import lightning_attn
    t = [torch.ones(1, 2, 64, 16) for _ in range(3)] + [torch.zeros(2, 1, 1)]
    if grad:
        t[(which + 1) % 3].requires_grad_(True)
    with fa.dual_level():
        t[which] = fa.make_dual(t[which], torch.ones_like(t[which]))
        with pytest.raises(NotImplementedError):
            lightning_attn(*t)
        with torch.no_grad(), pytest.raises(NotImplementedError):
            lightning_attn(*t)
