"""The work that users of this package have it do, as cases for timing: forward attention with Q/K RMSNorm and
rotary embedding through the public entry points, from one short prompt to the largest prefill batch.

A case is a dict of plain values:
  entry    "op"        ``optimized_attention`` on contiguous [B,H,S,D] tensors
           "layer"     ``fused`` on the [B,S,H,D] outputs of a model's projections, read in place, result written
                       as [B,S,Hq*D] for the output projection
           "factored"  ``factored_attention`` (no rotary embedding, query weight folded into the keys)
           "host"      ``optimized_attention_host`` on pinned CPU tensors
  B, S, Hq, Hkv, D     sizes;  dtype "bf16" / "fp16";  causal;  rope;  norm "hf" / "legacy";  theta
"""
import math

import torch

import kernelfuser_b200 as kf
from kernelfuser_b200.inputs import rope_tables

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}

# Query elements and operations of the largest cases (batch 16 at S = 4096 with 32 heads; the wide-head batch).
_MAX_Q = 1 << 28
_MAX_OPS = 4.4e12
# A host call moves its tensors over PCIe: its sizes stay where one call is a few milliseconds.
_MAX_Q_HOST = 1 << 25


def _case(entry, B, S, Hq, Hkv, D, dtype, causal=True, rope=True, norm="hf", theta=1e6):
    return {"entry": entry, "B": B, "S": S, "Hq": Hq, "Hkv": Hkv, "D": D, "dtype": dtype, "causal": causal,
            "rope": rope, "norm": norm, "theta": theta}


def listed():
    def named(name, *a, **kw):
        return {"name": name, **_case(*a, **kw)}

    return [
        # one short prompt of a 32/8-head model: launches and latency are what a user waits for
        named("prompt_128", "op", 1, 128, 32, 8, 128, "bf16"),
        # one ordinary prompt
        named("prompt_2k", "op", 1, 2048, 32, 8, 128, "bf16"),
        # a batch whose length is no multiple of any tile, in fp16
        named("ragged_fp16", "op", 4, 1000, 32, 8, 128, "fp16"),
        # prefill throughput: the headline batch
        named("prefill_4k", "op", 16, 4096, 32, 8, 128, "bf16"),
        # one long document
        named("document_16k", "op", 1, 16384, 32, 8, 128, "bf16"),
        # one rank's share of the headline batch when it is split by KV head over eight GPUs
        named("shard_of_8", "op", 16, 4096, 4, 1, 128, "bf16"),
        # wide heads, one short ragged prompt
        named("wide_1k_fp16", "op", 1, 1025, 16, 8, 256, "fp16", theta=1e4),
        # wide heads, the large batch
        named("wide_8k", "op", 8, 8192, 16, 8, 256, "bf16", theta=1e4),
        # inside a decoder layer: projections read in place, output written for the next projection
        named("layer_2k", "layer", 4, 2048, 32, 8, 128, "bf16"),
        # an encoder: no mask, no rotary embedding, as many KV heads as query heads, odd length
        named("encoder_1025", "op", 8, 1025, 8, 8, 128, "bf16", causal=False, rope=False, norm="legacy"),
        # the factored form for models with Q/K norm and no rotary embedding
        named("factored_2k", "factored", 4, 2048, 32, 8, 128, "bf16", rope=False, norm="legacy"),
        # tensors that live in host memory: copies and kernels of one call
        named("host_2k", "host", 4, 2048, 32, 8, 128, "bf16"),
    ]


def _pairs(S, causal):
    """(query, key) pairs of one head that the result depends on."""
    return S * (S + 1) // 2 if causal else S * S


def _ops(c):
    return 4.0 * c["B"] * c["Hq"] * _pairs(c["S"], c["causal"]) * c["D"]


def draw(rng):
    entry = rng.choice(["op", "op", "op", "op", "layer", "layer", "factored", "host"])
    D = 256 if entry != "factored" and rng.random() < 0.25 else 128
    # whole models, one rank's share of them, and heads without sharing
    Hq, Hkv = rng.choice([(16, 8), (8, 4), (4, 2), (2, 1)] if D == 256 else
                         [(32, 8), (32, 8), (16, 4), (8, 2), (4, 1), (8, 8), (8, 1)])
    causal = rng.random() < 0.8
    rope = entry != "factored" and rng.random() < 0.85
    norm = "legacy" if not rope else "hf"
    S = int(round(math.exp(rng.uniform(math.log(64), math.log(16384)))))
    if rng.random() < 0.5:  # half of the lengths are multiples of 128, the others as they come
        S = max(128, S // 128 * 128)
    B = int(round(math.exp(rng.uniform(0.0, math.log(16)))))
    c = _case(entry, B, S, Hq, Hkv, D, rng.choice(["bf16", "bf16", "fp16"]), causal, rope, norm,
              1e4 if D == 256 else 1e6)
    limit = _MAX_Q_HOST if entry == "host" else _MAX_Q
    while c["B"] > 1 and (c["B"] * Hq * S * D > limit or _ops(c) > _MAX_OPS):
        c["B"] -= 1
    while c["B"] * Hq * c["S"] * D > limit or _ops(c) > _MAX_OPS:
        c["S"] = c["S"] * 3 // 4
    return c


def prepare(case, seed):
    dtype = _DTYPES[case["dtype"]]
    B, S, Hq, Hkv, D = (case[n] for n in ("B", "S", "Hq", "Hkv", "D"))
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device=dev, dtype=dtype)

    if case["entry"] == "layer":  # the projections' outputs, as a model views them
        q, k, v = (normal(B, S, h * D).view(B, S, h, D).transpose(1, 2) for h in (Hq, Hkv, Hkv))
    else:
        q, k, v = (normal(B, h, S, D) for h in (Hq, Hkv, Hkv))
    gq, gk = ((1 + 0.1 * torch.randn(D, generator=gen, device=dev)).to(dtype) for _ in range(2))
    cos = sin = None
    if case["rope"]:
        cos, sin = rope_tables(torch.arange(S, device=dev), D, case["theta"], dtype)
        if case["entry"] == "layer":  # a model hands its tables on as [1,S,D]
            cos, sin = cos[None], sin[None]
    if case["entry"] == "host":
        q, k, v = (torch.empty(t.shape, dtype=dtype, pin_memory=True).copy_(t) for t in (q, k, v))
    state = {"case": case, "in": (q, k, v, gq, gk, cos, sin)}
    if case["entry"] == "host":
        state["out"] = torch.empty(q.shape, dtype=dtype, pin_memory=True)
    return state


def run(state):
    c = state["case"]
    q, k, v, gq, gk, cos, sin = state["in"]
    if c["entry"] == "op":
        return kf.optimized_attention(q, k, v, gq, gk, cos, sin, causal=c["causal"], norm_style=c["norm"])
    if c["entry"] == "layer":
        return kf.fused(q, k, v, gq, gk, cos, sin, c["causal"], norm_style=c["norm"], out_layout="bshd")
    if c["entry"] == "factored":
        return kf.factored_attention(q, k, v, gq, gk, causal=c["causal"])
    return kf.optimized_attention_host(q, k, v, gq, gk, cos, sin, causal=c["causal"], norm_style=c["norm"],
                                       out=state["out"])


def work(case):
    B, S, Hq, Hkv, D = (case[n] for n in ("B", "S", "Hq", "Hkv", "D"))
    values = 2 * B * S * D * (Hq + Hkv) + 2 * D + (2 * S * D if case["rope"] else 0)
    return {"bytes": 2 * values, "flops": _ops(case)}


def tolerance(case):
    # Measured on all listed and some drawn cases, as (norm of the difference, largest difference), against the
    # same path in 64 bits from its own prepared 16-bit rows and against another kernel of this package with its
    # sums in another order: bf16 up to 2.9e-3 and 5.1e-2, fp16 up to 3.7e-4 and 3.5e-3 (rounding the exact
    # result to the type already costs 1.6e-3 and 2.0e-4; the rest is the rounding of the probabilities).
    # Four times that:
    return {"rel": 1e-2, "max": 0.2} if case["dtype"] == "bf16" else {"rel": 1.5e-3, "max": 1.5e-2}


def exact(case, seed):
    """What ``run`` returns for these inputs, in 64 bits and without an intermediate rounding."""
    dev = torch.device("cuda", torch.cuda.current_device())
    q, k, v, gq, gk, cos, sin = (None if t is None else t.to(dev) for t in prepare(case, seed)["in"])
    B, S, Hq, Hkv, D = (case[n] for n in ("B", "S", "Hq", "Hkv", "D"))
    if cos is not None:
        cos, sin = cos.reshape(S, D).double(), sin.reshape(S, D).double()

    def rows(x, gamma):
        x = x.double()
        y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * gamma.double()
        if cos is None:
            return y
        lo, hi = y[..., : D // 2], y[..., D // 2:]
        return y * cos + torch.cat((-hi, lo), -1) * sin

    out = torch.empty(B, Hq, S, D, dtype=torch.float64, device=dev)
    step = max(1, min(S, (1 << 28) // S))  # query rows at a time: 2 GB of scores
    for b in range(B):
        for h in range(Hq):
            g = h // (Hq // Hkv)
            if h % (Hq // Hkv) == 0:
                kt, vv = rows(k[b, g], gk).t(), v[b, g].double()
            qn = rows(q[b, h], gq) * D ** -0.5
            for r in range(0, S, step):
                n = min(step, S - r)
                keys = r + n if case["causal"] else S  # later keys are masked for all of these rows
                s = qn[r: r + n] @ kt[:, :keys]
                if case["causal"]:
                    s.masked_fill_(torch.ones(n, keys, dtype=torch.bool, device=dev).triu_(r + 1), -math.inf)
                out[b, h, r: r + n] = torch.softmax(s, -1) @ vv
    return out.transpose(1, 2).reshape(B, S, Hq * D) if case["entry"] == "layer" else out
