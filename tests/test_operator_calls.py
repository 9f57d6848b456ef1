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
