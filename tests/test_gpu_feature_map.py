"""elu(x) + 1 of q and k ahead of the kernels (large calls) or inside them (small ones)."""
import pytest
import torch

from oracle import lasp_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 2, 16391, 128, 128), (2, 2, 16500, 64, 64), (1, 4, 8193, 128, 64)])
@pytest.mark.parametrize("scale,decay", [(1.0, False), (0.125, True)])
def test_feature_map_in_a_pass_of_its_own(shape, scale, decay):
    """From 2^22 elements of q on elu(x) + 1 is applied ahead of the kernels, below tile by tile inside them: both against the
    closed form in blocks, at lengths whose last tile has 7, 116 and 1 tokens.  A change to q before the backward pass is
    still noticed."""
    from lasp_b200 import lightning_attn_fused
    b, h, n, d, e = shape
    q, k, v, do = (t.to(torch.bfloat16) for t in O.make_inputs(n, b, h, n, d, e, scale_qk=False))
    s = O.baseline_slopes(h) if decay else torch.zeros(h, 1, 1)
    for rows in (n, 500):
        x = [t[:, :, :rows].contiguous() for t in (q, k, v, do)]
        ref = O.fwd_bwd_preprocessed(*(t.float() for t in x[:3]), s, x[3].float(), scale, "elu1")
        dev = [t.to("cuda:0").requires_grad_(i < 3) for i, t in enumerate(x)]
        o = lightning_attn_fused(*dev[:3], s.to("cuda:0"), qk_scale=scale, feature_map="elu1")
        with torch.no_grad():
            alone = lightning_attn_fused(*dev[:3], s.to("cuda:0"), qk_scale=scale, feature_map="elu1")
        assert O.max_rel_err(alone.float().cpu(), ref[0]) < 2e-2
        got = (o, *torch.autograd.grad(o, dev[:3], dev[3], retain_graph=True))
        for t, w, key in zip(got, ref, ("o", "dq", "dk", "dv")):
            assert O.max_rel_err(t.detach().float().cpu(), w) < 2e-2, (key, rows)
        with torch.no_grad():
            dev[0].zero_()
        with pytest.raises(RuntimeError, match="modified"):
            torch.autograd.grad(o, dev[:3], dev[3])


@pytest.mark.parametrize("shape", [(1, 160, 512, 64, 64), (2, 80, 300, 128, 128), (1, 4, 4099, 256, 256)])
@pytest.mark.parametrize("scale,decay", [(1.0, False), (0.125, True)])
def test_mapped_input_in_one_span_and_in_slices(shape, scale, decay):
    """More sequences than multiprocessors (a span each, several items a CTA), and 256-wide heads, whose slices read the mapped
    tensors in place and add their results up.  The oracle on the first and the last head, which nothing else enters."""
    from lasp_b200 import lightning_attn_fused
    b, h, n, d, e = shape
    q, k, v, do = (t.to(torch.bfloat16) for t in O.make_inputs(n, b, h, n, d, e, scale_qk=False))
    s = O.baseline_slopes(h) if decay else torch.zeros(h, 1, 1)
    dev = [t.to("cuda:0").requires_grad_(i < 3) for i, t in enumerate((q, k, v, do))]
    o = lightning_attn_fused(*dev[:3], s.to("cuda:0"), qk_scale=scale, feature_map="elu1")
    got = (o, *torch.autograd.grad(o, dev[:3], dev[3]))
    pick = [0, h - 1]
    ref = O.fwd_bwd_preprocessed(*(t[:, pick].float() for t in (q, k, v)), s[pick], do[:, pick].float(), scale, "elu1")
    for t, w, key in zip(got, ref, ("o", "dq", "dk", "dv")):
        assert O.max_rel_err(t[:, pick].detach().float().cpu(), w) < 2e-2, key


def test_what_a_large_folded_call_saves():
    """q and k once, mapped; under saved-tensor hooks, whose copies are their own, a later change is accepted as ever, and the
    gradients are those of the call."""
    from lasp_b200 import lightning_attn_fused
    b, h, n, d = 1, 4, 8200, 128
    q, k, v, do = (t.to("cuda:0", torch.bfloat16) for t in O.make_inputs(5, b, h, n, d, d, scale_qk=False))
    s = O.baseline_slopes(h).to("cuda:0")
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    want = torch.autograd.grad(lightning_attn_fused(*leaves, s, feature_map="elu1"), leaves, do)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(t), t.cpu())[1], lambda t: t.to("cuda:0")):
        o = lightning_attn_fused(*leaves, s, feature_map="elu1")
    assert sum(t.dtype == torch.bfloat16 for t in packed) == 3
    assert not any(t.data_ptr() == x.data_ptr() for t in packed for x in leaves[:2])
    with torch.no_grad():
        leaves[0].zero_(), leaves[1].zero_()
    for a, w in zip(torch.autograd.grad(o, leaves, do), want):
        assert torch.equal(a, w)
    with torch.inference_mode():
        qi = q.clone()
    with pytest.raises(RuntimeError, match="Inference tensors cannot be saved"):
        lightning_attn_fused(qi, k, leaves[2], s, feature_map="elu1")
