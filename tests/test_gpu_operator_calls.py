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


def _gradients_through(pack, unpack, n=200):
    from lasp_b200 import lightning_attn
    q, k, v = (t.requires_grad_(True) for t in _inputs(4, n))
    s = torch.full((2, 1, 1), 0.01, device=DEV)
    plain = torch.autograd.grad(lightning_attn(q, k, v, s), (q, k, v), torch.ones_like(v))
    with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
        o = lightning_attn(q, k, v, s)
    return plain, torch.autograd.grad(o, (q, k, v), torch.ones_like(v))


@pytest.mark.parametrize("n", [100, 200])
def test_saved_tensors_may_come_back_laid_out_differently(n):
    """A hook that transposes, offloads or changes the type of the decay rates: same gradients."""
    def back(t):
        if t.dim() == 4:
            return t.transpose(2, 3).contiguous().transpose(2, 3)      # the values in another order in memory
        return t.double().cpu() if t.dtype == torch.float32 else t
    for pack, unpack in ((lambda t: t, back), (lambda t: t.cpu(), lambda t: t.to(DEV))):
        plain, got = _gradients_through(pack, unpack, n)
        for a, b in zip(plain, got):
            assert torch.equal(a, b)


@pytest.mark.parametrize("change", [lambda t: t.half(), lambda t: t.cpu(), lambda t: t[..., :32], lambda t: t[:, :, 1:]])
def test_saved_tensors_that_are_not_what_they_were_are_refused(change):
    """... and one that changes what it was given is told so, before anything is launched."""
    for kind in (4, 1):                                                 # q, k, v; the states kept by the forward pass
        def back(t):
            if t.dim() != kind or (kind == 1 and t.dtype != torch.uint8):
                return t
            return change(t.view(1, 1, 1, -1) if kind == 1 else t)
        with pytest.raises((RuntimeError, TypeError, ValueError), match="saved"):
            _gradients_through(lambda t: t, back)


def test_calls_on_several_streams_at_once():
    """Threads with a stream each: the CTAs of their launches share the SMs, every launch has its own synchronisation words,
    and the results are those of the calls one after the other."""
    import threading
    from lasp_b200 import engine, lightning_attn
    shapes = [(2, 12, 2048, 128), (1, 40, 1500, 64), (1, 4, 4096, 128)]

    def inputs(i, rep):
        b, h, n, d = shapes[i]
        g = torch.Generator(device=DEV).manual_seed(100 * i + rep)
        t = [torch.randn(b, h, n, d, generator=g, device=DEV).to(torch.bfloat16) for _ in range(4)]
        return [x.requires_grad_(j < 3) for j, x in enumerate(t)], torch.full((h, 1, 1), 0.002, device=DEV)

    def call(t, s):
        o = lightning_attn(*t[:3], s)
        return [o.detach(), *torch.autograd.grad(o, t[:3], t[3])]

    sets = [[inputs(i, rep) for rep in range(4)] for i in range(len(shapes))]
    want = [[call(*x) for x in s] for s in sets]
    got = [[None] * 12 for _ in shapes]
    torch.cuda.synchronize()

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for k in range(12):
                got[i][k] = call(*sets[i][k % 4])
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(shapes))]
    [t.start() for t in threads], [t.join() for t in threads]
    assert engine.read_status() == 0
    for i in range(len(shapes)):
        for k in range(12):
            for a, b in zip(got[i][k], want[i][k % 4]):
                assert torch.equal(a, b), (shapes[i], k)
