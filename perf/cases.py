"""The work whose speed counts: calls of the public operators as training and inference programs make them.

A case is one operator call on one GPU: a forward pass (``op`` "forward"), or a forward and a backward pass
(``op`` "train"), through ``lightning_attn``, ``lightning_attn_fused`` (the preprocessing of q and k inside the
kernels) or ``lasp_fuse_parallel`` (a rank whose sequence-parallel group is itself alone).  Shapes are
(b, h, n, d) for q and k and (b, h, n, e) for v.
"""
import math

import torch

import lasp_b200
from lasp_b200.utils import build_slope_tensor, initialize_lasp, sequence_parallel_is_initialized

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _case(name, entry, op, dtype, b, h, n, d, e, decay=True, elu=False):
    c = dict(entry=entry, op=op, dtype=dtype, b=b, h=h, n=n, d=d, e=e, decay=decay, elu=elu)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a short prompt through one narrow layer: the smallest call, host time and launches
        _case("forward_small", "lightning", "forward", "bf16", 1, 8, 256, 64, 64),
        # a rank of a purely data-parallel job that keeps the sequence-parallel operator in its model (the DP x 1
        # rows of the reference's comparison), at the reference test's shape
        _case("dp_rank", "fuse_parallel", "train", "bf16", 2, 12, 2048, 128, 64),
        # the headline training layer
        _case("train_headline", "lightning", "train", "bf16", 2, 12, 2048, 128, 128),
        # a training batch of packed documents: length not a multiple of any tile
        _case("train_ragged", "lightning", "train", "bf16", 3, 12, 3001, 128, 128),
        # many sequences of ordinary length, more than the chip has multiprocessors
        _case("train_batch", "lightning", "train", "bf16", 8, 32, 2048, 128, 128),
        # one rank's share of a long sequence, 16 heads
        _case("train_share", "lightning", "train", "bf16", 1, 16, 16384, 128, 128),
        # the whole 131072-token sequence on one GPU: the largest
        _case("train_long", "lightning", "train", "bf16", 1, 16, 131072, 128, 128),
        # prefill of a long prompt, 32 heads
        _case("prefill", "lightning", "forward", "bf16", 1, 32, 16384, 128, 128),
        # no decay, elu(x) + 1 on q and k inside the kernels, 64-wide heads
        _case("nodecay_folded", "lightning_fused", "train", "bf16", 4, 16, 4096, 64, 64, decay=False, elu=True),
        # the same configuration with 256-wide heads, q and k mapped by the caller
        _case("nodecay_wide", "lightning", "train", "bf16", 4, 16, 4096, 256, 256, decay=False),
        # fp32 training at the headline shape (the parity configuration)
        _case("train_fp32", "lightning", "train", "fp32", 2, 12, 2048, 128, 128),
        # fp16 training (autocast) at the reference test's shape
        _case("train_fp16", "lightning", "train", "fp16", 2, 12, 2048, 128, 64),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """The ranges: 1-8 batch rows, 2-40 heads, 64-131072 tokens (any number), head widths of 64 and 128 in every
    combination, sometimes 96 or 256; bf16 mostly, fp16 and fp32 at up to the headline's number of tokens."""
    dtype = rng.choices(["bf16", "fp16", "fp32"], [70, 15, 15])[0]
    entry = rng.choices(["lightning", "lightning_fused", "fuse_parallel"], [70, 15, 15])[0]
    op = "train" if rng.random() < 0.7 else "forward"
    d, e = rng.choices([(128, 128), (128, 64), (64, 128), (64, 64), (96, 96), (256, 256)], [40, 15, 5, 20, 10, 10])[0]
    if entry == "lightning_fused":
        dtype = "bf16"
    if dtype != "bf16" and d == 256:
        d = e = 128
    h = rng.choice([2, 4, 8, 12, 12, 16, 16, 20, 24, 32, 32, 40])
    b = rng.choice([1, 1, 2, 2, 3, 4, 6, 8])
    # tokens x heads of the whole call, in units of 128-wide heads
    most = (1 << 20 if dtype == "bf16" else 49152) * 256 / (d + e) / (2 if d > 128 else 1)
    if d == 96 and dtype == "bf16":
        most = 49152
    n = _log_uniform(rng, 64, max(128, min(131072, most / (b * h))))
    if rng.random() < 0.4 and n >= 256:
        n = n // 128 * 128
    elu = entry == "lightning_fused"
    # (without decay the sums of a long sequence leave fp16's range)
    return _case(None, entry, op, dtype, b, h, n, d, e, decay=rng.random() < 0.8 or dtype == "fp16", elu=elu)


def prepare(case, seed):
    b, h, n, d, e = (case[x] for x in ("b", "h", "n", "d", "e"))
    dtype = DTYPES[case["dtype"]]
    device = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=device).manual_seed(int(seed))

    def normal(width):
        return torch.randn(b, h, n, width, generator=g, device=device)

    q, k = normal(d), normal(d)
    if case["decay"]:
        s = build_slope_tensor(h).to(device)
        if not case["elu"]:
            q, k = q * d ** -0.5, k * d ** -0.5
    else:
        s = torch.zeros(h, 1, 1, device=device)
        if not case["elu"]:   # the caller maps q and k
            q, k = torch.nn.functional.elu(q) + 1.0, torch.nn.functional.elu(k) + 1.0
    train = case["op"] == "train"
    state = {"case": case, "s": s, "train": train}
    for name, t in (("q", q), ("k", k), ("v", normal(e))):
        state[name] = t.to(dtype).requires_grad_(train)
    if train:
        state["do"] = normal(e).to(dtype)
    if case["entry"] == "fuse_parallel":
        if not torch.distributed.is_initialized():
            torch.distributed.init_process_group("nccl", store=torch.distributed.HashStore(), rank=0, world_size=1)
        if not sequence_parallel_is_initialized():
            initialize_lasp(1, 1)
        state["KV"] = torch.empty(b, h, d, e, device=device)
        state["DKV"] = torch.empty(b, h, d, e, device=device)
    return state


def run(state):
    case = state["case"]
    q, k, v, s = state["q"], state["k"], state["v"], state["s"]
    if case["entry"] == "lightning":
        o = lasp_b200.lightning_attn(q, k, v, s)
    elif case["entry"] == "lightning_fused":
        scale = case["d"] ** -0.5 if case["decay"] else 1.0
        o = lasp_b200.lightning_attn_fused(q, k, v, s, qk_scale=scale, feature_map="elu1" if case["elu"] else None)
    else:
        o = lasp_b200.lasp_fuse_parallel(q, k, v, s, state["KV"], state["DKV"])
    if not state["train"]:
        return {"o": o}
    dq, dk, dv = torch.autograd.grad(o, (q, k, v), state["do"])
    return {"o": o.detach(), "dq": dq, "dk": dk, "dv": dv}


def work(case):
    """Every input read once and every output written once; the arithmetic of the recurrence, which no blocked
    form undercuts: state update and read-out forward (4 d e per token and head), twice that backward."""
    b, h, n, d, e = (case[x] for x in ("b", "h", "n", "d", "e"))
    tokens, size = b * h * n, DTYPES[case["dtype"]].itemsize
    moved, flops = 2 * d + 2 * e, 4 * d * e
    if case["op"] == "train":
        moved, flops = moved + 4 * d + 3 * e, flops * 3   # q, k, v, do read, dq, dk, dv written
    return {"bytes": tokens * moved * size + 4 * h, "flops": tokens * flops}


def tolerance(case):
    """bf16 and fp16 round the results to 8 and 11 bits (bf16 intermediates too); fp32 sums differ in their order."""
    return {"rel": {"bf16": 1e-2, "fp16": 2e-3, "fp32": 1e-5}[case["dtype"]]}
