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


@pytest.mark.parametrize("dtype,gate", [(torch.float32, 3e-6), (torch.float16, 2e-3), (torch.bfloat16, 1e-2)])
@pytest.mark.parametrize("shape", [(1, 2, 1, 16, 16), (2, 1, 64, 48, 96), (1, 2, 65, 96, 112), (1, 3, 130, 128, 80), (2, 2, 300, 80, 128)])
def test_rank_states_in_and_out(dtype, gate, shape):
    """Border states travel as three bf16 terms; lengths of up to 64 tokens are where the workspace has the least room for
    them.  Gates: the type's rounding of results, 3e-6 for the fp32 states of every type."""
    from lasp_b200 import engine
    b, h, n, d, e = shape
    q, k, v, do = (t.to(dtype) for t in O.make_inputs(800 + n + d, b, h, n, d, e))
    s = torch.tensor([0.0, 0.03, 1.0][:h])
    gen = torch.Generator().manual_seed(n)
    kv_in, dkv_in = (torch.randn(b, h, d, e, generator=gen) for _ in range(2))
    plan = engine.make_plan(b, h, n, d, e, dtype)
    guard = 4096
    spaces = [torch.full((plan.ws_bytes + 2 * guard,), 0x5A, dtype=torch.uint8, device=DEV) for _ in range(2)]
    ws = [x[guard:guard + plan.ws_bytes] for x in spaces]
    qd, kd, vd, dod, sd = (t.to(DEV) for t in (q, k, v, do, s))
    kv_out, dkv_out = (torch.empty(b, h, d, e, device=DEV) for _ in range(2))
    fw = engine.Forward(plan, qd, kd, vd, sd, kv_in=kv_in.to(DEV), kv_out=kv_out, ws=ws[0])
    o = fw.run()
    bw = engine.Backward(plan, qd, kd, vd, dod, sd, fw.ws, dkv_in=dkv_in.to(DEV), dkv_out=dkv_out, ws=ws[1])
    got = (o, *bw.run())
    wide = [t.double() for t in (q, k, v)]
    ref_o, ref_kv = O.blocked_forward(*wide, s, kv_in.double(), dtype=torch.float64)
    ref = O.blocked_backward(*wide, s, do.double(), kv_in.double(), dkv_in.double(), dtype=torch.float64)
    for t, w, key in zip(got, (ref_o, *ref[:3]), ("o", "dq", "dk", "dv")):
        assert O.max_rel_err(t.double().cpu(), w) < gate, key
    assert O.max_rel_err(kv_out.double().cpu(), ref_kv) < 3e-6
    assert O.max_rel_err(dkv_out.double().cpu(), ref[3]) < 3e-6
    for x in spaces:
        assert bool((x[:guard] == 0x5A).all()) and bool((x[-guard:] == 0x5A).all())
    assert engine.read_status() == 0


@pytest.mark.parametrize("dtype,gate", [(torch.float32, 3e-6), (torch.bfloat16, 1e-2)])
def test_exchange_scan_of_the_full_precision_path(dtype, gate):
    """Two ranks of a sequence, one launch after the other on one GPU: what the first stores for the second is in its slots
    when its launch begins, so nothing waits."""
    from lasp_b200 import _cabi, engine
    b, h, n, d, e = 2, 2, 200, 96, 80
    q, k, v, _ = (t.to(dtype) for t in O.make_inputs(900, b, h, 2 * n, d, e))
    s = torch.tensor([0.0, 0.02])
    sd = s.to(DEV)
    plan = engine.make_plan(b, h, n, d, e, dtype)
    new = lambda words: torch.zeros(words, dtype=torch.int32, device=DEV)
    slots = [new(2 * 2 * b * h * d * e * 2) for _ in range(2)]
    acks = [new(2 * 8 * 32) for _ in range(2)]
    outs = []
    for r in range(2):
        part = [t[:, :, r * n:(r + 1) * n].contiguous().to(DEV) for t in (q, k, v)]
        fw = engine.Forward(plan, *part, sd)
        fw.chunk_states()
        a = _cabi.ExchangeArgs()
        counters = new(64)
        a.ranks, a.position, a.reverse = 2, r, 0
        a.s, a.ws, a.ws_bytes = sd.data_ptr(), fw.ws.data_ptr(), fw.ws.numel()
        a.my_slots, a.my_acks, a.counters = slots[r].data_ptr(), acks[r].data_ptr(), counters.data_ptr()
        for i in range(2):
            a.peer_slots[i], a.peer_acks[i] = slots[i].data_ptr(), acks[i].data_ptr()
        engine.exchange_scan(plan, a, torch.device(DEV))
        fw.output()
        outs.append(fw.o)
        torch.cuda.synchronize()
    ref = O.blocked_forward(*(t.double() for t in (q, k, v)), s, dtype=torch.float64)[0]
    assert O.max_rel_err(torch.cat(outs, 2).double().cpu(), ref) < gate
    assert engine.read_status() == 0
