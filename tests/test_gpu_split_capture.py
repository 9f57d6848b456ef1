"""The full-precision kernels' launches follow on one another by programmatic serialisation: captured into a graph, with a
branch of another stream joined right before the first of them, a step gives the bits of an eager one on whatever the
inputs hold at replay."""
import pytest
import torch

from oracle import lasp_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype,width", [(torch.float32, 128), (torch.float16, 64), (torch.bfloat16, 96)])
@pytest.mark.parametrize("n", [100, 700])
def test_captured_step_replays_as_an_eager_one(dtype, width, n):
    from lasp_b200 import engine, lightning_attn
    b, h = 2, 4
    s = O.baseline_slopes(h).to(DEV)
    draws = [[t.to(DEV, dtype) for t in O.make_inputs(seed, b, h, n, width, width)] for seed in (1, 2, 3)]
    q, k, v, do = (t.clone().requires_grad_(i < 3) for i, t in enumerate(draws[0]))
    raw = draws[0][3].clone()

    def step():
        o = lightning_attn(q, k, v, s)
        return (o, *torch.autograd.grad(o, (q, k, v), do))

    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(3):
            step()
    side.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        other.wait_stream(side)
        with torch.cuda.stream(other):
            do.copy_(raw)
        side.wait_stream(other)
        captured = step()
    for x in draws[1:] + draws[:1]:
        with torch.no_grad():
            for t, new in zip((q, k, v), x):
                t.copy_(new)
            raw.copy_(x[3])
        graph.replay()
        torch.cuda.synchronize()
        got = [t.detach().clone() for t in captured]
        for a, w, key in zip(got, step(), ("o", "dq", "dk", "dv")):
            assert torch.equal(a, w.detach()), key
    assert engine.read_status() == 0
    del captured, graph
