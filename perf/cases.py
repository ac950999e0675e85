"""Performance cases of the fused-MoE path: what a serving or evaluation program has it do.

A case is a dict of plain values; ``listed()`` gives the named ones, ``draw(rng)`` one more of the same
ranges.  ``prepare`` makes what a program holds before the call (activations, routing, expert weights),
``run`` is one pass through the public entry points, ``work`` what the pass cannot do without.

Kinds:
  int4    ``fused_moe_int4_w4a16``: one grouped expert GEMM of an INT4 layer with its top-k combine
  ffn     ``fused_moe_int4_ffn``: the whole two-GEMM INT4 expert layer
  mxfp4   ``fused_moe_mxfp4``: the whole MXFP4 expert layer
  ep      the expert side of one expert-parallel rank: received rows -> partial rows
          (``moe_int4_w4a16_partial``) and the owner's sum of a token's partials (``moe_gather_sum_reduce``)
  router  ``topk_softmax``
  align   ``moe_align_block_size``
  reduce  ``moe_sum_reduce``
"""

from __future__ import annotations

import torch

import xkernels_b200 as xkb
from xkernels_b200 import ops, synth

_DT = {"bf16": torch.bfloat16, "fp32": torch.float32, "fp16": torch.float16}
_ESIZE = {"bf16": 2, "fp32": 4, "fp16": 2}


def _int4(M, K, N, E, top_k, group=32, skew=0.0, **name):
    return dict(name, kind="int4", M=M, K=K, N=N, E=E, top_k=top_k, group=group, skew=skew)


def listed():
    return [
        # one sequence decoding: eight experts' weights, launches and latency count
        _int4(1, 7168, 4096, 48, 8, name="int4_gate_up_m1"),
        # the headline: a decode batch, every expert hit by a handful of tokens, weight streaming
        _int4(64, 7168, 4096, 48, 8, name="int4_gate_up_m64"),
        # a speculative or mixed batch of an odd size through the layer's second GEMM shape
        _int4(509, 2048, 7168, 48, 8, name="int4_down_m509"),
        # prefill with mildly skewed routing: tensor-pipe bound, the largest case
        _int4(16384, 7168, 4096, 48, 8, skew=0.5, name="int4_gate_up_m16384"),
        # the other common group size of 4-bit checkpoints, decode batch
        _int4(64, 7168, 4096, 48, 8, group=128, name="int4_g128_m64"),
        # the whole INT4 expert layer in one call, decode batch of an odd size
        dict(name="int4_ffn_m37", kind="ffn", M=37, hidden=7168, inter=2048, E=48, top_k=8, skew=0.0),
        # the MXFP4 expert layer: decode, many experts with one or two tokens each
        dict(name="mxfp4_m48", kind="mxfp4", M=48, hidden=4096, ispp=512, E=256, top_k=6, bias=False),
        # the MXFP4 expert layer: prefill chunk, with the biases that such layers may have
        dict(name="mxfp4_m4096", kind="mxfp4", M=4096, hidden=4096, ispp=512, E=256, top_k=6, bias=True),
        # one rank of an eight-rank expert-parallel layer in a prefill step
        dict(name="ep_rank_r6144", kind="ep", R=6144, M=1024, K=7168, N=2048, E=32, top_k=8, world=8),
        # the router of a prefill step
        dict(name="router_m16384", kind="router", M=16384, E=256, topk=8, dtype="bf16", renorm=True),
        # the routing sort of a prefill step, without a host read (what a serving loop uses)
        dict(name="align_m16384", kind="align", M=16384, top_k=8, E=48, block=16),
        # the top-k combine of a prefill step on its own
        dict(name="reduce_m8192", kind="reduce", M=8192, top_k=8, H=7168, dtype="bf16"),
    ]


def _log_int(rng, lo, hi):
    """log-uniform integer in [lo, hi]; odd ones as likely as even ones"""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def _skew(rng):
    """spread of the experts' popularity (logit bias), from none to strong"""
    return round(0.8 * rng.random(), 3)


_MOST_FLOPS = 2.0 * 16384 * 8 * 4096 * 7168


def draw(rng):
    u = rng.random()
    if u < 0.40:
        # the two GEMM shapes of the INT4 layer, a smaller layer, the expert-parallel shape; group 128 now and then
        K, N, E, top_k = rng.choice([(7168, 4096, 48, 8), (7168, 4096, 48, 8), (2048, 7168, 48, 8),
                                     (4096, 2048, 64, 6), (7168, 2048, 256, 8)])
        group = 128 if rng.random() < 0.15 else 32
        # group 128 is drawn up to mid-sized batches
        M = _log_int(rng, 1, 512 if group != 32 else 16384)
        M = max(1, min(M, int(_MOST_FLOPS / (2.0 * top_k * N * K))))
        return _int4(M, K, N, E, top_k, group=group, skew=_skew(rng))
    if u < 0.55:
        hidden, inter, E, top_k = rng.choice([(7168, 2048, 48, 8), (7168, 2048, 48, 8), (4096, 1024, 64, 6)])
        return dict(kind="ffn", M=_log_int(rng, 1, 4096), hidden=hidden, inter=inter, E=E, top_k=top_k,
                    skew=_skew(rng))
    if u < 0.75:
        hidden, ispp, E, top_k = rng.choice([(4096, 512, 256, 6), (4096, 512, 256, 6), (4096, 1024, 128, 4),
                                             (2048, 1024, 64, 6)])
        return dict(kind="mxfp4", M=_log_int(rng, 1, 8192), hidden=hidden, ispp=ispp, E=E, top_k=top_k,
                    bias=rng.random() < 0.3)
    if u < 0.82:
        world = rng.choice([2, 4, 8])
        R = _log_int(rng, 64, 16384)
        return dict(kind="ep", R=R, M=max(1, R // 6), K=7168, N=2048, E=256 // world, top_k=8, world=world)
    if u < 0.88:
        return dict(kind="router", M=_log_int(rng, 1, 65536), E=rng.choice([48, 64, 128, 256, 384]),
                    topk=rng.choice([4, 6, 8]), dtype=rng.choice(["bf16", "bf16", "fp32", "fp16"]),
                    renorm=rng.random() < 0.7)
    if u < 0.94:
        E, top_k = rng.choice([(48, 8), (64, 6), (256, 8), (256, 6)])
        return dict(kind="align", M=_log_int(rng, 1, 32768), top_k=top_k, E=E,
                    block=rng.choice([16, 32, 64, 128]))
    return dict(kind="reduce", M=_log_int(rng, 1, 16384), top_k=rng.choice([4, 6, 8]),
                H=rng.choice([2048, 4096, 7168]), dtype=rng.choice(["bf16", "bf16", "fp32"]))


def _seed(case, seed):
    return int(seed) * 1009 + 17


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    s = _seed(case, seed)
    kind = case["kind"]
    if kind == "int4":
        A = synth.activations(case["M"], case["K"], seed=s, device=dev)
        packed, scale = synth.int4_weights(case["E"], case["N"], case["K"], case["group"], seed=s + 1, device=dev)
        ids, w = synth.routing(case["M"], case["E"], case["top_k"], seed=s + 3, device=dev, expert_bias_std=case["skew"])
        return dict(kind=kind, A=A, packed=packed, scale=scale, ids=ids, w=w, group=case["group"])
    if kind == "ffn":
        A = synth.activations(case["M"], case["hidden"], seed=s, device=dev)
        w13, s13 = synth.int4_weights(case["E"], 2 * case["inter"], case["hidden"], 32, seed=s + 1, device=dev)
        w2, s2 = synth.int4_weights(case["E"], case["hidden"], case["inter"], 32, seed=s + 5, device=dev)
        # per-layer weight magnitudes of about 1/sqrt(fan-in), so that the hidden activations are O(1)
        s13, s2 = s13 * 0.125, s2 * 0.25
        ids, w = synth.routing(case["M"], case["E"], case["top_k"], seed=s + 3, device=dev, expert_bias_std=case["skew"])
        return dict(kind=kind, A=A, w13=w13, s13=s13, w2=w2, s2=s2, ids=ids, w=w)
    if kind == "mxfp4":
        A = synth.activations(case["M"], case["hidden"], seed=s, device=dev)
        # scale bytes around 2^-7: weights of about 1/sqrt(fan-in)
        wts = synth.mxfp4_weights(case["E"], case["hidden"], case["ispp"], seed=s + 1, device=dev, scale_lo=117,
                                  scale_hi=121, with_bias=case["bias"])
        ids, w = synth.routing(case["M"], case["E"], case["top_k"], seed=s + 3, device=dev)
        return dict(kind=kind, A=A, wts=wts, ids=ids, w=w)
    if kind == "ep":
        R, k, E = case["R"], case["top_k"], case["E"]
        g = torch.Generator(device=dev).manual_seed(s)
        A = synth.activations(R, case["K"], seed=s + 1, device=dev)
        packed, scale = synth.int4_weights(E, case["N"], case["K"], 32, seed=s + 2, device=dev)
        # a received row has at least one of its top-k slots on this rank, each slot with chance 1 / world
        here = torch.rand(R, k, generator=g, device=dev) < 1.0 / case["world"]
        here[:, 0] |= ~here.any(dim=1)
        ids, w = synth.routing(R, E, k, seed=s + 4, device=dev, expert_bias_std=0.5)
        ids = torch.where(here, ids, torch.full_like(ids, -1))
        w = torch.where(here, w, torch.zeros_like(w))
        routing = torch.cat([ids, w.view(torch.int32)], dim=1).contiguous()
        # each own token's partials: some of the rows (their positions are known from the plan)
        index = torch.randint(0, R, (case["M"], case["world"]), generator=g, device=dev, dtype=torch.int32)
        index[torch.rand(case["M"], case["world"], generator=g, device=dev) < 0.35] = -1
        return dict(kind=kind, A=A, packed=packed, scale=scale, routing=routing, index=index)
    if kind == "router":
        g = torch.Generator(device=dev).manual_seed(s)
        x = torch.randn(case["M"], case["E"], generator=g, device=dev, dtype=torch.float32).to(_DT[case["dtype"]])
        return dict(kind=kind, x=x, topk=case["topk"], renorm=case["renorm"])
    if kind == "align":
        ids, _ = synth.routing(case["M"], case["E"], case["top_k"], seed=s, device=dev, expert_bias_std=0.5)
        return dict(kind=kind, ids=ids, block=case["block"], E=case["E"])
    if kind == "reduce":
        g = torch.Generator(device=dev).manual_seed(s)
        y = torch.randn(case["M"], case["top_k"], case["H"], generator=g, device=dev, dtype=torch.float32)
        w = torch.softmax(torch.randn(case["M"], case["top_k"], generator=g, device=dev), dim=-1)
        return dict(kind=kind, y=y.to(_DT[case["dtype"]]), w=w)
    raise ValueError(f"unknown kind {kind!r}")


def run(state):
    kind = state["kind"]
    if kind == "int4":
        return xkb.fused_moe_int4_w4a16(state["A"], state["packed"], state["scale"], state["ids"], state["w"],
                                        group_size=state["group"])
    if kind == "ffn":
        return xkb.fused_moe_int4_ffn(state["A"], state["w13"], state["s13"], state["w2"], state["s2"], state["ids"],
                                      state["w"])
    if kind == "mxfp4":
        t = state["wts"]
        return xkb.fused_moe_mxfp4(state["A"], t["w13"], t["w13_scale"], t["w2"], t["w2_scale"], state["ids"], state["w"],
                                   b13=t["b13"], b2=t["b2"])
    if kind == "ep":
        rows = ops.moe_int4_w4a16_partial(state["A"], state["packed"], state["scale"], state["routing"])
        return rows, ops.moe_gather_sum_reduce(rows, state["index"], None)
    if kind == "router":
        return xkb.topk_softmax(state["x"], state["topk"], state["renorm"])
    if kind == "align":
        return xkb.moe_align_block_size(state["ids"], state["block"], state["E"], truncate=False)
    if kind == "reduce":
        return xkb.moe_sum_reduce(state["y"], state["w"])
    raise ValueError(f"unknown kind {kind!r}")


def _int4_rows64(A, packed, scale, group, tok, ids, E, N):
    """[slots, N] float64: A[tok] @ W[ids]^T; the weight is what the format says, code x scale rounded to bf16"""
    shifts = 4 * torch.arange(8, device=A.device, dtype=torch.int32)
    out = torch.zeros(ids.numel(), N, dtype=torch.float64, device=A.device)
    for e in range(E):
        at = (ids == e).nonzero(as_tuple=True)[0]
        if at.numel() == 0:
            continue
        codes = ((packed[e].unsqueeze(-1) >> shifts) & 15).reshape(N, -1) - 8
        W = (codes.float() * scale[e].float().repeat_interleave(group, dim=1)).to(torch.bfloat16).double()
        out[at] = A[tok[at]].double() @ W.t()
    return out


def _silu_up64(gate, up, limit):
    if limit:
        gate, up = gate.clamp(max=limit), up.clamp(-limit, limit)
    return gate * torch.sigmoid(gate) * up


def _mx64(w, scale, e):
    """[rows, K] float64 weights of expert e: E2M1 codes (low nibble = even k) x 2^(byte - 127)"""
    table = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6, -0.0, -0.5, -1, -1.5, -2, -3, -4, -6], dtype=torch.float64,
                         device=w.device)
    codes = torch.stack([w[e] & 15, w[e] >> 4], dim=-1).reshape(w.shape[1], -1)
    return table[codes.long()] * torch.exp2(scale[e].double() - 127).repeat_interleave(32, dim=1)


def _combine64(rows, w, M, top_k):
    return (rows * w.reshape(-1, 1).double()).reshape(M, top_k, -1).sum(dim=1)


def exact(case, seed):
    """``run``'s outputs in 64 bits from plain torch.  Weights are what their formats say; no other rounding."""
    st = prepare(case, seed)
    kind = case["kind"]
    if kind == "align":
        return None
    if kind == "router":
        p = torch.softmax(st["x"].double(), dim=-1)
        w = torch.topk(p, st["topk"], dim=-1).values
        return (w / w.sum(dim=-1, keepdim=True) if st["renorm"] else w), None
    if kind == "reduce":
        return torch.cat([(y.double() * w.double().unsqueeze(-1)).sum(dim=1)
                          for y, w in zip(st["y"].split(1024), st["w"].split(1024))])
    if kind == "ep":
        R, k = case["R"], case["top_k"]
        ids, w = st["routing"][:, :k].reshape(-1), st["routing"][:, k:].contiguous().view(torch.float32)
        tok = torch.arange(R, device=ids.device).repeat_interleave(k)
        rows = _combine64(_int4_rows64(st["A"], st["packed"], st["scale"], 32, tok, ids, case["E"], case["N"]), w, R, k)
        at = st["index"].long()
        return rows, (rows[at.clamp(min=0)] * (at >= 0).unsqueeze(-1)).sum(dim=1)
    ids, w, M, k = st["ids"].reshape(-1), st["w"], case["M"], case["top_k"]
    tok = torch.arange(M, device=ids.device).repeat_interleave(k)
    if kind == "int4":
        out = torch.zeros(M, case["N"], dtype=torch.float64, device=ids.device)
        step = max(1, 65536 // k)
        for lo in range(0, M, step):
            hi = min(M, lo + step)
            s = slice(lo * k, hi * k)
            rows = _int4_rows64(st["A"], st["packed"], st["scale"], st["group"], tok[s], ids[s], case["E"], case["N"])
            out[lo:hi] = _combine64(rows, w[lo:hi], hi - lo, k)
        return out
    if kind == "ffn":
        I = case["inter"]
        gu = _int4_rows64(st["A"], st["w13"], st["s13"], 32, tok, ids, case["E"], 2 * I)
        act = _silu_up64(gu[:, :I], gu[:, I:], 0.0)
        slot = torch.arange(M * k, device=ids.device)
        return _combine64(_int4_rows64(act, st["w2"], st["s2"], 32, slot, ids, case["E"], case["hidden"]), w, M, k)
    if kind == "mxfp4":
        t, I = st["wts"], case["ispp"]
        rows = torch.zeros(M * k, case["hidden"], dtype=torch.float64, device=ids.device)
        for e in range(case["E"]):
            at = (ids == e).nonzero(as_tuple=True)[0]
            if at.numel() == 0:
                continue
            gu = st["A"][tok[at]].double() @ _mx64(t["w13"], t["w13_scale"], e).t()
            if t["b13"] is not None:
                gu = gu + t["b13"][e].double()
            down = _silu_up64(gu[:, :I], gu[:, I:], 10.0) @ _mx64(t["w2"], t["w2_scale"], e).t()
            rows[at] = down if t["b2"] is None else down + t["b2"][e].double()
        return _combine64(rows, w, M, k)
    raise ValueError(f"unknown kind {kind!r}")


def _active(E, slots):
    """experts hit by `slots` slots, each token's distinct"""
    return min(E, E * (1.0 - (1.0 - 1.0 / E) ** slots))


def work(case):
    kind = case["kind"]
    if kind == "int4":
        M, K, N, k = case["M"], case["K"], case["N"], case["top_k"]
        act = k if M == 1 else _active(case["E"], M * k)
        return {"bytes": act * N * (K / 2 + 2 * K / case["group"]) + 2 * M * (K + N) + 8 * M * k,
                "flops": 2.0 * M * k * N * K}
    if kind == "ffn":
        M, H, I, k = case["M"], case["hidden"], case["inter"], case["top_k"]
        act = k if M == 1 else _active(case["E"], M * k)
        return {"bytes": act * 3 * H * I * (1 / 2 + 2 / 32) + 4 * M * H + 8 * M * k, "flops": 6.0 * M * k * H * I}
    if kind == "mxfp4":
        M, H, I, k = case["M"], case["hidden"], case["ispp"], case["top_k"]
        act = k if M == 1 else _active(case["E"], M * k)
        return {"bytes": act * 3 * H * I * (1 / 2 + 1 / 32) + 4 * M * H + 8 * M * k, "flops": 6.0 * M * k * H * I}
    if kind == "ep":
        R, K, N, k = case["R"], case["K"], case["N"], case["top_k"]
        p = 1.0 / case["world"]
        slots = R * (k * p + (1.0 - p) ** k)          # at least one slot per row is here
        act = _active(case["E"], slots)
        return {"bytes": act * N * (K / 2 + 2 * K / 32) + R * (2 * K + 4 * N + 8 * k)
                + 0.65 * case["M"] * case["world"] * 4 * N + 2 * case["M"] * N, "flops": 2.0 * slots * N * K}
    if kind == "router":
        return {"bytes": case["M"] * (case["E"] * _ESIZE[case["dtype"]] + 8 * case["topk"]), "flops": 0}
    if kind == "align":
        n = case["M"] * case["top_k"]
        pad = n + (case["E"] + 1) * (case["block"] - 1)
        return {"bytes": 4 * (n + pad + pad // case["block"] + 1), "flops": 0}
    if kind == "reduce":
        e = _ESIZE[case["dtype"]]
        return {"bytes": case["M"] * ((case["top_k"] + 1) * case["H"] * e + 4 * case["top_k"]), "flops": 0}
    raise ValueError(f"unknown kind {kind!r}")


def tolerance(case):
    """About four times what the tensor-core path and the generic path (the same roundings, sums in another
    order) were seen to differ by; the router and the bare reduce against sums in 64 bits."""
    kind = case["kind"]
    if kind == "align":
        return "exact"
    if kind == "router":
        # seen 7e-8; ids may only differ where two probabilities tie
        return {"rel": 3e-7, "differ": 1e-4}
    if kind == "reduce":
        # bf16: flips of the final rounding (a rounding alone is 1.7e-3 of the exact sum)
        return {"rel": 1e-3} if case["dtype"] == "bf16" else {"rel": 1e-6}
    if kind == "ffn":
        return {"rel": 4e-3}      # seen 1.1e-3: three bf16 roundings on the way
    if kind == "mxfp4":
        return {"rel": 1.5e-3}    # seen 3.3e-4
    return {"rel": 8e-4}          # int4, ep: seen 2e-4, flips of the final bf16 rounding
