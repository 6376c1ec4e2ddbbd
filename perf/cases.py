"""The timed cases of the MoE expert layer: what a serving process has this library do, through the entry points of
`hecate_b200.moe` that such a process calls.

A case is one layer call. `flow` names the calls it makes:

    decode    router_decode + moe4_combine: a decode step of a layer whose experts are all on this GPU (the benchmark's step)
    normed    norm_route + decode + combine_norm: the same step where the residual add and the input norms are fused into it
    band      decode on a selection made elsewhere, this GPU holding a band [lo, lo + n) of the router's experts
    forward   forward on given selections: prompt chunks of any length; the library picks the kernels by the row count
    router    router_fused alone (a prompt chunk's routing)

The other keys are the layer (H, I, experts = router positions, local = experts held here from `lo` on, group = columns per weight
scale, 0 = one fp32 scale per row, shared = format of the shared expert), the rows, the activation type and the skew of the
routing (Zipf exponent of the experts' popularity, 0 = uniform). The mode that reproduces the CPU engine's int8 activation
round trips is a parity check, not a mode of operation, and has no case.
"""
import math

import torch

from hecate_b200 import moe

TOPK = 8
FULL = dict(H=6144, I=2048, experts=256)       # the benchmark's layer: 4.85 GB of int4 experts


def case(flow, rows, layer=FULL, local=None, lo=0, group=128, shared="int4", act="bf16", zipf=0.0):
    return dict(flow=flow, rows=rows, **layer, local=layer["experts"] if local is None else local, lo=lo, group=group, shared=shared,
                act=act, zipf=zipf)


def listed():
    named = lambda name, *a, **k: dict(name=name, **case(*a, **k))
    return [
        # a single user's token: latency of the launch chain and 9 experts' bytes
        named("decode-1", "decode", 1),
        # a smaller layer at a few rows: hardly any bytes, so launches and host work count
        named("decode-4-small-layer", "decode", 4, dict(H=2048, I=768, experts=64)),
        # the reference's own weight format (fp32 row scales, int8 shared expert, fp16 rows), step with both norms fused
        named("decode-8-row-scales-normed", "normed", 8, group=0, shared="int8", act="fp16"),
        # one rank of four, or one processor of several: a quarter of the experts, foreign picks ignored
        named("decode-11-band", "band", 11, local=64, lo=128, shared="none"),
        # the benchmark's decode step: 8 sequences with one draft token each
        named("decode-16", "decode", 16),
        # a layer wider than the benchmark's
        named("decode-6-wide-layer", "decode", 6, dict(H=7168, I=2560, experts=64)),
        # short prompt chunks, or decode steps of many sequences
        named("forward-48", "forward", 48),
        named("forward-200-row-scales", "forward", 200, group=0, shared="int8", act="fp16"),
        # a ragged chunk between short prompts and full chunks, skewed routing
        named("forward-777-skewed", "forward", 777, zipf=1.1),
        # a chunk in the reference's format, routed experts only
        named("forward-2048-row-scales", "forward", 2048, group=0, shared="none", act="fp16"),
        # the benchmark's prefill chunk
        named("forward-8192-skewed", "forward", 8192, zipf=1.1),
        # and the routing of such a chunk
        named("router-8192", "router", 8192),
    ]


def draw(rng):
    flow = rng.choice(["decode", "decode", "normed", "band", "forward", "forward", "forward", "forward", "router"])
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    if rng.random() < 0.5:
        layer = dict(FULL)
    else:
        # generic layers of up to the benchmark's weight per expert, those wider than it in either direction in steps of 1024
        # columns; the norm and router kernels take H % 256 == 0
        while True:
            layer = dict(H=256 * rng.randint(4, 32), I=128 * rng.randint(4, 24), experts=32 * rng.randint(1, 8))
            wide = layer["H"] > 6144 or layer["I"] > 2048
            if layer["H"] * layer["I"] <= FULL["H"] * FULL["I"] and (flow != "normed" or layer["H"] <= 6144) and (not wide or layer["H"] % 1024 == 0):
                break
    n = layer["experts"]
    local, lo = n, 0
    if flow == "band" or (flow == "forward" and rng.random() < 0.2):
        local = max(8, n // rng.choice([2, 4, 8]))
        lo = rng.randrange(0, n - local + 1)
    rows = {"decode": rng.randint(1, 16), "normed": rng.randint(1, 16), "band": rng.randint(1, 16), "router": log(1, 8192)}.get(flow) or log(17, 8192)
    # the int8 shared expert's decode kernels take layers of up to 6144 x 2048
    shared = rng.choice(["int4", "int4", "int8", "none"] if layer["H"] <= 6144 and layer["I"] <= 2048 else ["int4", "none"])
    return case(flow, rows, layer, local, lo, group=rng.choice([0, 128]), shared=shared, act=rng.choice(["bf16", "fp16"]),
                zipf=rng.choice([0.0, 0.7, 1.1, 1.3]) if flow in ("band", "forward") else 0.0)


class State:
    """The layer's weights, router and buffers, and one batch of rows."""


def _experts(s, c, seed, gen, dev):
    H, I, n, group = c["H"], c["I"], c["local"], c["group"]
    per = H * I // 2
    total = n + (c["shared"] == "int4")
    pool = torch.empty(total * 3 * per, dtype=torch.uint8, device=dev)
    moe.fill_bytes(pool, seed, 1)                               # uniform int4 codes
    w = pool.view(total, 3, per)
    # scales lognormal(-4, 0.5), in the order the kernels read them
    lognormal = lambda *shape: (torch.randn(*shape, device=dev, generator=gen) * 0.5 - 4.0).exp()
    if group:
        scales = [lognormal(total, N // 64, K // group, 64).to(torch.bfloat16) for N, K in ((I, H), (I, H), (H, I))]
    else:
        scales = [lognormal(total, N) for N in (I, I, H)]
    shared = None
    if c["shared"] == "int4":
        shared = (w[n, 0], w[n, 1], w[n, 2], scales[0][n], scales[1][n], scales[2][n])
    elif c["shared"] == "int8":
        q = torch.empty(3, H * I, dtype=torch.uint8, device=dev)
        moe.fill_bytes(q, seed, 2)
        shared = (q[0], q[1], q[2], *(lognormal(N) / 16 for N in (I, I, H)))
    s.tables = moe.ExpertTables(H, I, TOPK, list(w[:n, 0]), list(w[:n, 1]), list(w[:n, 2]), list(scales[0][:n]), list(scales[1][:n]),
                                list(scales[2][:n]), group=group, shared=shared, device=dev, shared_i8=c["shared"] == "int8")


def prepare(c, seed):
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed + 1)
    R, H, I, E, flow = c["rows"], c["H"], c["I"], c["experts"], c["flow"]
    dtype = torch.bfloat16 if c["act"] == "bf16" else torch.float16
    s = State()
    s.flow, s.rows, s.lo = flow, R, c["lo"]
    s.x = torch.randn(R, H, device=dev, generator=gen).to(torch.bfloat16).to(dtype)
    s.sel = torch.zeros(R, TOPK, dtype=torch.int64, device=dev)
    s.rw = torch.zeros(R, TOPK, dtype=torch.float16, device=dev)
    if flow in ("decode", "normed", "router"):
        s.wt = (torch.randn(E, H, device=dev, generator=gen) * 0.02).to(torch.bfloat16).to(dtype)
        s.bias = torch.randn(E, device=dev, generator=gen) * 0.02
    else:
        # top-8 without replacement from the experts' popularity, positive weights that sum to one
        logp = -c["zipf"] * torch.log(torch.arange(1, E + 1, device=dev, dtype=torch.float32))
        u = torch.rand(R, E, device=dev, generator=gen).clamp_(1e-7, 1 - 1e-7)
        s.sel.copy_((logp - torch.log(-torch.log(u))).topk(TOPK, dim=1).indices)
        w = torch.rand(R, TOPK, device=dev, generator=gen) + 0.05
        s.rw.copy_(w / w.sum(1, keepdim=True))
    if flow == "router":
        return s
    _experts(s, c, seed, gen, dev)
    zeros = lambda: torch.zeros(R, H, dtype=torch.float32, device=dev)
    s.out = zeros()
    if flow == "forward":
        s.ws = moe.forward_workspace(R, TOPK, c["local"], H, I, dev)
        return s
    s.ws = moe.decode_workspace(H, I, dev)
    if flow == "decode":
        s.acc = zeros()
    elif flow == "normed":
        s.acc, s.resid, s.o = zeros(), torch.randn(R, H, device=dev, generator=gen), torch.randn(R, H, device=dev, generator=gen)
        s.norms = [(1 + 0.1 * torch.randn(H, device=dev, generator=gen)).to(dtype) for _ in range(2)]
        s.xn = [torch.zeros(R, H, dtype=torch.float16, device=dev) for _ in range(2)]
    return s


def run(s):
    if s.flow == "decode":
        s.out.zero_()
        moe.router_decode(s.tables, s.x, s.wt, s.bias, s.sel, s.rw, 1.0, s.acc, s.ws)
        moe.moe4_combine(s.out, 0, s.acc, s.rows, 0)
        return s.out, s.sel, s.rw
    if s.flow == "normed":
        # s.out carries the residual: the attention output s.o joins it in front, the experts' output behind
        moe.norm_route(s.o, s.resid, s.norms[0], s.xn[0], s.wt, s.bias, s.sel, s.rw, TOPK, 1.0, 1e-5, r_out=s.out)
        moe.decode(s.tables, s.xn[0], s.sel, s.rw, s.acc, s.ws)
        moe.combine_norm(None, 0, s.acc, s.rows, 0, 0, s.out, s.norms[1], s.xn[1], 1e-5)
        return s.out, s.xn[0], s.xn[1], s.sel, s.rw
    if s.flow == "band":
        s.out.zero_()
        return moe.decode(s.tables, s.x, s.sel, s.rw, s.out, s.ws, lo=s.lo)
    if s.flow == "forward":
        s.out.zero_()
        return moe.forward(s.tables, s.x, s.sel, s.rw, s.out, s.ws, lo=s.lo)
    moe.router_fused(s.x, s.wt, s.bias, None, None, s.sel, s.rw, TOPK, 1.0)
    return s.sel, s.rw


def _inclusion(c):
    """Probability that a row picks each expert (sampling without replacement as exponential races: 1 - exp(-rate p))."""
    p = [(e + 1.0) ** -c["zipf"] for e in range(c["experts"])]
    lo, hi = 0.0, 1.0
    picks = lambda rate: sum(1 - math.exp(-rate * v) for v in p)
    while picks(hi) < TOPK:
        hi *= 2
    for _ in range(60):
        mid = (lo + hi) / 2
        lo, hi = (mid, hi) if picks(mid) < TOPK else (lo, mid)
    return [1 - math.exp(-hi * v) for v in p]


def work(c):
    R, H, I, E, flow = c["rows"], c["H"], c["I"], c["experts"], c["flow"]
    routing = R * TOPK * (8 + 2)
    nbytes, flops = R * H * 2 + routing, 0.0
    if flow in ("decode", "normed", "router"):
        nbytes += E * H * 2 + E * 4
        flops += 2.0 * R * E * H
    if flow == "router":
        return {"bytes": float(nbytes), "flops": flops}
    held = _inclusion(c)[c["lo"]:c["lo"] + c["local"]]
    picks = R * sum(held)
    distinct = sum(1 - (1 - q) ** R for q in held)
    expert = 3 * H * I // 2 + ((2 * I * H + H * I) // c["group"] * 2 if c["group"] else (2 * I + H) * 4)
    nbytes += distinct * expert + R * H * 4
    if flow == "normed":
        nbytes += R * H * (4 + 2) + 2 * H * 2                  # the attention output, the second normalised copy, the norm weights
    if c["shared"] != "none":
        nbytes += expert if c["shared"] == "int4" else 3 * H * I + (2 * I + H) * 4
        picks += R
    return {"bytes": float(nbytes), "flops": flops + picks * 6.0 * H * I}


def tolerance(c):
    if c["flow"] == "router":
        return "exact"                                          # selections and fp16 weights are reproducible bit for bit
    # fp16 operands, fp32 sums: against the same layer in 64 bits the listed cases are off by 1.8e-4 to 2.8e-4 (largest single value
    # 0.8e-3 to 2.6e-3), nearly all of it the one rounding of the SiLU product; another implementation rounds it elsewhere
    return {"rel": 1e-3, "max": 1e-2}
