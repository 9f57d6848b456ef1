"""The fused launches that hand the rank state over themselves (lasp_b200_forward_linked, lasp_b200_bwd_dkv_linked), one rank
at a time on one GPU: what the ranks before it would have stored is put into its slots by the host, and what it stores
for the ranks after it goes to ordinary memory, where the test reads it."""
import ctypes as C
import time

import pytest
import torch

from oracle import lasp_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
ACK = 32     # acknowledgement words: (position * 8) * 32


def _words(states, step):
    """(b,h,d,e) states as the {value, step} words of one source's slot: per float4 of a row two planes of 16 bytes."""
    b, h, d, e = states.shape
    w = states.float().reshape(b, h, d, e // 4, 2, 2).permute(0, 1, 3, 4, 2, 5).contiguous()
    return torch.stack([w.view(torch.int32), torch.full_like(w, step, dtype=torch.int32)], -1).reshape(-1)


def _states(words, shape):
    b, h, d, e = shape
    w = words.reshape(-1, 2)[:, 0].contiguous().view(torch.float32)
    return w.reshape(b, h, e // 4, 2, d, 2).permute(0, 1, 4, 2, 3, 5).reshape(b, h, d, e)


class Rank:
    """The peer-mapped buffers of one rank at place `pos` of `ranks` in the chain order of one direction."""

    def __init__(self, ranks, pos, shape, step, wait_clocks=0):
        from lasp_b200 import _cabi
        self.ranks, self.pos, self.shape, self.step = ranks, pos, shape, step
        self.elems = shape[0] * shape[1] * shape[2] * shape[3]
        new = lambda n: torch.zeros(n, dtype=torch.int32, device=DEV)
        self.slots = new(2 * ranks * self.elems * 2)
        self.peer_slots = [new(2 * ranks * self.elems * 2) for _ in range(ranks)]
        self.acks, self.peer_acks, self.counters = new(8 * 8 * ACK), [new(8 * 8 * ACK) for _ in range(ranks)], new(64)
        self.counters[0] = step - 1
        self.acks += max(step - 2, 0)                 # the readers are done with the slots' use before the last
        self.args = a = _cabi.ExchangeArgs()
        a.ranks, a.position, a.wait_clocks = ranks, pos, wait_clocks
        a.my_slots, a.my_acks, a.counters = self.slots.data_ptr(), self.acks.data_ptr(), self.counters.data_ptr()
        for i in range(ranks):
            a.peer_slots[i], a.peer_acks[i] = self.peer_slots[i].data_ptr(), self.peer_acks[i].data_ptr()

    def slot(self, buf, source):
        at = ((self.step & 1) * self.ranks + source) * self.elems * 2
        return buf[at:at + self.elems * 2]

    def check_sent(self, total, reach):
        """total: what this rank sends; reach(hops): heads whose state gets there."""
        for dst in range(self.ranks):
            got = self.slot(self.peer_slots[dst], self.pos)
            if dst <= self.pos:
                assert not got.any()
                continue
            heads = reach(dst - self.pos - 1)
            got = got.reshape(self.shape[0], self.shape[1], -1).cpu()
            assert bool((got[:, heads].reshape(-1, 2)[:, 1] == self.step).all()) and not got[:, ~heads].any()
            part = (self.shape[0], int(heads.sum()), *self.shape[2:])
            if part[1]:
                assert O.max_rel_err(_states(got[:, heads].reshape(-1), part), total[:, heads]) < 1e-2
        for src in range(self.ranks):
            assert self.peer_acks[src][self.pos * 8 * ACK].item() == (self.step if src < self.pos else 0)
        assert self.counters[0].item() == self.step


class Problem:
    """A rank's chunk in the middle of a sequence whose other chunks are there as their totals only."""

    def __init__(self, ranks, pos, b, n, d, e, slopes, scale=1.0, fmap=None, seed=0):
        from lasp_b200 import engine
        h = len(slopes)
        self.s, self.n, self.pos, self.ranks, self.scale, self.fmap = torch.tensor(slopes).reshape(h, 1, 1), n, pos, ranks, scale, fmap
        q, k, v, do = O.make_inputs(seed + n, b, h, n, d, e, scale_qk=fmap is None and scale == 1.0)
        self.x = [t.to(torch.bfloat16) for t in (q, k, v, do)]
        self.dev = [t.to(DEV) for t in self.x]
        g = torch.Generator().manual_seed(seed + 1)
        self.other = [torch.randn(b, h, d, e, generator=g) for _ in range(ranks)]       # totals of the other ranks
        self.shape = (b, h, d, e)
        self.sn = self.s.reshape(-1) * n
        extra = dict(qk_scale=scale, feature_map=fmap) if (fmap or scale != 1.0) else {}
        self.plan = engine.make_plan(b, h, n, d, e, torch.bfloat16, **extra)
        assert engine.linked_ok(self.plan)

    def reach(self, hops):
        return self.sn * hops <= 27.6

    def incoming(self, place):
        """the state that arrives at `place` of the chain order"""
        acc = torch.zeros(self.shape, dtype=torch.float64)
        for src in range(place):
            hops = place - 1 - src
            acc += (torch.exp(-self.sn.double() * hops) * self.reach(hops)).reshape(1, -1, 1, 1) * self.other[src]
        return acc

    def fill(self, rank):
        for src in range(rank.pos):
            w = _words(self.other[src], rank.step).reshape(self.shape[0], self.shape[1], -1)
            w[:, ~self.reach(rank.pos - 1 - src)] = 0          # is not sent: nobody may wait for it
            rank.slot(rank.slots, src).copy_(w.reshape(-1))

    def expected(self):
        """o, total, dq, dk, dv, backward total; the rank is at `pos` forward and at ranks-1-pos backward"""
        q, k, v, do = (t.double() for t in self.x)
        mq, mk = (O.preprocess_qk(t, self.scale, self.fmap) for t in (q, k))
        kv_in, dkv_in = self.incoming(self.pos), self.incoming(self.ranks - 1 - self.pos)
        o, _ = O.blocked_forward(mq, mk, v, self.s, kv_in, dtype=torch.float64)
        _, total = O.blocked_forward(mq, mk, v, self.s, None, dtype=torch.float64)
        dq, dk, dv, _ = O.blocked_backward(mq, mk, v, self.s, do, kv_in, dkv_in, dtype=torch.float64)
        *_, dtotal = O.blocked_backward(mq, mk, v, self.s, do, None, None, dtype=torch.float64)
        slope = [O.preprocess_slope(t, self.scale, self.fmap) for t in (q, k)]
        return o, total, dq * slope[0], dk * slope[1], dv, dtotal

    def forward(self, rank):
        from lasp_b200 import engine
        fw = engine.Forward(self.plan, *self.dev[:3], self.s)
        fw.run_linked(rank.args)
        return fw

    def backward(self, rank, fw):
        from lasp_b200 import engine
        q, k, v, do = self.dev
        bw = engine.Backward(self.plan, q, k, v, do, self.s, fw.ws)
        bw.dq_only()
        bw.dkv_linked(rank.args)
        return bw


SLOPES = [0.0, 0.002, 0.02, 1.5]        # reach every rank, every rank, the next one or two, the next rank only


@pytest.mark.parametrize("ranks,pos", [(2, 0), (2, 1), (4, 0), (4, 1), (4, 2), (4, 3)])
@pytest.mark.parametrize("d,e,n", [(128, 128, 1000), (128, 64, 2048), (64, 128, 700), (64, 64, 3001)])
@pytest.mark.parametrize("scale,fmap", [(1.0, None), (0.125, "elu1")])
def test_a_rank_of_a_group(ranks, pos, d, e, n, scale, fmap):
    from lasp_b200 import engine
    p = Problem(ranks, pos, 2, n, d, e, SLOPES, scale, fmap)
    o, total, dq, dk, dv, dtotal = p.expected()
    for step in (1, 6):                                # the first hand-over, and one whose slots have been used before
        fr = Rank(ranks, pos, p.shape, step)
        p.fill(fr)
        fw = p.forward(fr)
        br = Rank(ranks, ranks - 1 - pos, p.shape, step)
        p.fill(br)
        bw = p.backward(br, fw)
        torch.cuda.synchronize()
        assert engine.read_status() == 0
        for got, want, key in ((fw.o, o, "o"), (bw.dq, dq, "dq"), (bw.dk, dk, "dk"), (bw.dv, dv, "dv")):
            assert O.max_rel_err(got.float(), want) < 2e-2, (key, step)
        fr.check_sent(total, p.reach)
        br.check_sent(dtotal, p.reach)


def test_a_late_peer_is_waited_for():
    """The words of the rank before arrive more than half a second - the limit of every other wait of the kernels - after
    the launch: same results, no fault."""
    from lasp_b200 import engine
    p = Problem(2, 1, 1, 1000, 128, 128, [0.0, 0.01])
    o, total, dq, dk, dv, dtotal = p.expected()
    side = torch.cuda.Stream()
    limit = 6_000_000_000                                 # clocks: three seconds
    late, back = Rank(2, 1, p.shape, 1, limit), Rank(2, 1, p.shape, 1, limit)
    p.pos = 0                                             # (backward: the first rank of the sequence, last of the chain)
    dk0, dv0 = p.expected()[3:5]
    p.pos = 1
    words = _words(p.other[0], 1).pin_memory()
    torch.cuda.synchronize()
    for rank in (late, back):
        if rank is late:
            fw = p.forward(rank)
        else:
            bw = engine.Backward(p.plan, *p.dev, p.s, fw.ws)
            bw.dkv_linked(rank.args)
        time.sleep(1.0)
        with torch.cuda.stream(side):
            rank.slot(rank.slots, 0).copy_(words, non_blocking=True)
        torch.cuda.synchronize()
    assert engine.read_status() == 0
    for got, want in ((fw.o, o), (bw.dk, dk0), (bw.dv, dv0)):
        assert O.max_rel_err(got.float(), want) < 2e-2


def test_a_peer_that_never_delivers_is_reported():
    """The wait for it runs out after longer than the other waits' limit: its own bit of the fault word and no other, NaN
    where its state would have gone, right results in the head that it does not reach."""
    from lasp_b200 import engine
    p = Problem(3, 2, 1, 1000, 128, 128, [0.0, 0.01, 1.5])
    o = p.expected()[0]
    rank = Rank(3, 2, p.shape, 1, 1_500_000_000)
    p.fill(rank)
    rank.slot(rank.slots, 1).reshape(1, 3, -1)[:, :2] = 0      # heads 0 and 1 of the rank before are missing
    fw = p.forward(rank)
    torch.cuda.synchronize()
    assert engine.read_status() == 4
    assert bool(torch.isnan(fw.o[:, :2]).all())
    assert O.max_rel_err(fw.o[:, 2].float(), o[:, 2]) < 2e-2
    assert engine.read_status() == 0
