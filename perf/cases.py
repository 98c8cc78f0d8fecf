"""The calls whose speed this repository stands for: what a program that uses the operators has them do.

A case is a dict of plain values.  ``op`` names the public entry point:

* ``fwd``     ``miniattn.flash_attn_fwd`` (prefill, chunked prefill and decode; (B,H,N,D) or (B,N,H,D))
* ``compat``  ``miniattn.forward``, the drop-in operator of the reference ((B,N,H,D), non-causal)
* ``int8``    ``miniattn.flash_attn_fwd_int8qk`` with the pre-pass, on buffers the program keeps
* ``ring``    ``miniattn.parallel.ring_forward``: one rank's launches with the state carried between them
* ``shard``   ``miniattn.parallel.sharded_forward``: one rank's share of the (batch x KV head) units
* ``module``  ``miniattn.variants.GQA_Flash`` (projections + attention)

``Nq`` query rows are the last ``Nq`` of ``Nk`` positions where the call is causal.
"""
from __future__ import annotations

import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "mini-attention_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import miniattn  # noqa: E402
from miniattn import parallel, variants  # noqa: E402

_DT = {"fp16": torch.float16, "bf16": torch.bfloat16}


def _case(name, op, B, Hq, Hkv, Nq, Nk, D, dtype, causal=False, layout="bhnd", lse=False, world=1):
    c = {"op": op, "B": B, "Hq": Hq, "Hkv": Hkv, "Nq": Nq, "Nk": Nk, "D": D, "dtype": dtype, "causal": causal,
         "layout": layout, "lse": lse, "world": world}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # The reference's own correctness recipe through its drop-in operator: the smallest call, where
        # host time, launch and a work item's fixed cost count.
        _case("compat_n512", "compat", 2, 8, 8, 512, 512, 128, "fp16", layout="bnhd"),
        # The middle and the end of the N = 512..8192 sweep that the headline metric is quoted on.
        _case("mha_n2048", "fwd", 2, 8, 8, 2048, 2048, 128, "fp16"),
        _case("mha_n8192", "fwd", 2, 8, 8, 8192, 8192, 128, "fp16"),
        # Training / prefill of a grouped-query decoder, whole batch on one GPU ...
        _case("gqa_causal_n4096", "fwd", 4, 32, 8, 4096, 4096, 128, "bf16", causal=True),
        # ... and the share of it that one of eight GPUs computes.
        _case("gqa_shard8_n4096", "shard", 4, 32, 8, 4096, 4096, 128, "bf16", causal=True, world=8),
        # Head dim 64, causal, a batch of short sequences, with the log-sum-exp that a backward pass needs.
        _case("d64_causal_n1024", "fwd", 4, 12, 12, 1024, 1024, 64, "bf16", causal=True, lse=True),
        # Ragged lengths, an odd number of heads, head dim 96.
        _case("d96_ragged_n1001", "fwd", 3, 7, 7, 1001, 1001, 96, "fp16"),
        # Chunked prefill: the next 777 tokens of two requests against everything seen so far, three query
        # heads to a KV head, the (B,N,H,D) layout that projections produce, lse for a later merge.
        _case("chunk_prefill_777", "fwd", 2, 24, 8, 777, 3333, 128, "bf16", causal=True, layout="bnhd", lse=True),
        # Decode: one new token of 16 requests against a KV cache.
        _case("decode_b16_n4001", "fwd", 16, 32, 8, 1, 4001, 128, "bf16", causal=True),
        # INT8-QK: quantising pre-pass and attention, K with a per-channel offset.
        _case("int8qk_n8192", "int8", 2, 16, 16, 8192, 8192, 64, "fp16"),
        # The module: four projections around the attention call.
        _case("gqa_module_s1024", "module", 2, 16, 4, 1024, 1024, 128, "bf16", causal=True, layout="bnhd"),
        # Long context: the ring launcher on one GPU (three launches, the rows' state carried).
        _case("ring_n131072", "ring", 1, 32, 32, 131072, 131072, 128, "fp16", causal=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        op = rng.choice(["compat", "fwd", "fwd", "fwd", "chunk", "decode", "decode", "int8", "ring", "shard", "module"])
        dtype = rng.choice(["fp16", "bf16"])
        hkv = rng.choice([1, 2, 4, 5, 8, 16])
        g = rng.choice([1, 1, 2, 3, 4, 8])
        b = rng.choice([1, 1, 2, 3, 4, 8])
        layout = rng.choice(["bhnd", "bnhd"])
        lse = rng.random() < 0.3
        n = _log(rng, 128, 16384)
        if rng.random() < 0.4:
            n = max(128, n // 128 * 128)
        if op == "compat":
            n = max(64, n // 64 * 64)
            c = _case("", op, b, hkv, hkv, n, n, 128, "fp16", layout="bnhd")
        elif op == "fwd":
            c = _case("", op, b, hkv * g, hkv, n, n, rng.choice([64, 96, 128, 128]), dtype, rng.random() < 0.5, layout, lse)
        elif op == "chunk":
            c = _case("", "fwd", b, hkv * g, hkv, _log(rng, 16, 2048), n + 2048, rng.choice([64, 128, 128]), dtype, True,
                      layout, lse)
        elif op == "decode":
            c = _case("", "fwd", rng.choice([1, 2, 4, 8, 16, 32, 64]), hkv * g, hkv, rng.choice([1, 1, 1, 2, 4, 5]),
                      _log(rng, 300, 65536), rng.choice([64, 128, 128]), dtype, True, layout, lse)
        elif op == "int8":
            c = _case("", op, b, hkv * g, hkv, n, n, rng.choice([64, 64, 128]), dtype, rng.random() < 0.5)
        elif op == "ring":
            n = max(1024, n // 2 * 2)
            c = _case("", op, b, hkv, hkv, n, n, 128, dtype, True)
        elif op == "shard":
            c = _case("", op, b, hkv * g, hkv, n, n, 128, dtype, rng.random() < 0.7, world=rng.choice([2, 4, 8]))
            if b * hkv < c["world"]:
                continue
        else:
            n = min(n, 4096)
            if hkv * g > 32:
                continue
            c = _case("", "module", min(b, 4), hkv * g, hkv, n, n, rng.choice([64, 128]), dtype, True, "bnhd")
        w = work(c)
        if w["flops"] <= 4e12 and w["bytes"] <= 4e9:
            return c


def _normal(gen, shape, dtype):
    return torch.randn(shape, generator=gen, device="cuda", dtype=_DT[dtype])


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    B, Hq, Hkv, Nq, Nk, D, dt = c["B"], c["Hq"], c["Hkv"], c["Nq"], c["Nk"], c["D"], c["dtype"]
    if c["op"] == "module":
        d = Hq * D
        with torch.device("cuda"):
            m = variants.GQA_Flash(d, Hq, Hkv).to(_DT[dt]).requires_grad_(False)
        with torch.no_grad():
            for p in m.parameters():
                p.normal_(0.0, 1.0 / math.sqrt(d), generator=gen)
        return {"case": c, "m": m, "x": _normal(gen, (B, Nq, d), dt)}
    if c["layout"] == "bhnd":
        # K and V are the filled part of a cache with room for more tokens where the call is a decode or a chunk
        room = Nk if Nq == Nk else (Nk + 511) // 256 * 256
        q = _normal(gen, (B, Hq, Nq, D), dt)
        k, v = (_normal(gen, (B, Hkv, room, D), dt)[:, :, :Nk] for _ in range(2))
    else:
        room = Nk if Nq == Nk else (Nk + 511) // 256 * 256
        q = _normal(gen, (B, Nq, Hq, D), dt)
        k, v = (_normal(gen, (B, room, Hkv, D), dt)[:, :Nk] for _ in range(2))
    s = {"case": c, "q": q, "k": k, "v": v}
    if c["op"] == "int8":
        s["k"] = k + 2.0 * _normal(gen, (B, Hkv, 1, D), dt)
        s["buffers"] = miniattn.Int8QK(B, Hq, Hkv, Nq, Nk, D, q.device)
    if c["op"] == "shard":
        s["out"] = torch.zeros_like(q)
    return s


def run(state):
    c = state["case"]
    op = c["op"]
    if op == "module":
        return state["m"](state["x"])
    q, k, v = state["q"], state["k"], state["v"]
    if op == "compat":
        return miniattn.forward(q, k, v)
    if op == "int8":
        return miniattn.flash_attn_fwd_int8qk(q, k, v, causal=c["causal"], buffers=state["buffers"])
    if op == "ring":
        return parallel.ring_forward(q, k, v, causal=c["causal"])
    if op == "shard":
        return parallel.sharded_forward(q, k, v, causal=c["causal"], rank=0, world=c["world"], out=state["out"])
    return miniattn.flash_attn_fwd(q, k, v, causal=c["causal"], layout=c["layout"], return_lse=c["lse"],
                                   q_pos0=c["Nk"] - c["Nq"])


def work(case):
    c = case
    B, Hq, Hkv, Nq, Nk, D = c["B"], c["Hq"], c["Hkv"], c["Nq"], c["Nk"], c["D"]
    # (query, key) pairs of one head that the rule shows
    pairs = Nq * Nk - (Nq * (Nq - 1) // 2 if c["causal"] else 0)
    if c["op"] == "shard":
        units = len(parallel.shard_units(B, Hkv, c["world"], 0))
        B, Hq, Hkv = 1, units * (Hq // Hkv), units
    flops = 4.0 * B * Hq * pairs * D
    if c["op"] == "module":
        d, dkv = Hq * D, Hkv * D
        flops += 2.0 * B * Nq * d * (2 * d + 2 * dkv)
        return {"bytes": 2.0 * (2 * B * Nq * d + d * (2 * d + 2 * dkv) + 2 * d + 2 * dkv), "flops": flops}
    nbytes = 2.0 * B * D * (2 * Hq * Nq + 2 * Hkv * Nk)
    if c["lse"]:
        nbytes += 4.0 * B * Hq * Nq
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # Fp32 sums around a 16-bit P and 16-bit results.  Against the same formula in 64 bits the cases show
    # rel 2.9e-4 to 3.0e-4 in fp16 and 2.1e-3 to 2.6e-3 in bf16 (largest single difference 0.011 and 0.082 of the
    # root mean square); the bounds are four times that.
    return {"rel": 1.2e-3, "max": 0.045} if case["dtype"] == "fp16" else {"rel": 1e-2, "max": 0.33}


def _quantised(x):
    """int8 per block of 128 tokens and back: round-half-even(x / scale) * scale, scale = max|x| / 127 in fp32."""
    B, H, N, D = x.shape
    pad = (N + 127) // 128 * 128 - N
    blocks = torch.nn.functional.pad(x.float(), (0, 0, 0, pad)).view(B, H, -1, 128, D)
    scale = blocks.abs().amax((3, 4), keepdim=True) / 127.0
    scale = torch.where(scale > 0, scale, torch.ones_like(scale))
    q = (blocks / scale).round().clamp(-127, 127).double() * scale.double()
    return q.view(B, H, N + pad, D)[:, :, :N]


def _attention64(q, k, v, causal):
    """(B,H,N,D) -> fp64 output and log-sum-exp; causal rows are the last positions."""
    B, Hq, Nq, D = q.shape
    Hkv, Nk = k.shape[1], k.shape[2]
    out = torch.empty((B, Hq, Nq, D), dtype=torch.float64, device=q.device)
    lse = torch.empty((B, Hq, Nq), dtype=torch.float64, device=q.device)
    step = max(1, (1 << 26) // Nk)
    cols = torch.arange(Nk, device=q.device)
    for b in range(B):
        for h in range(Hq):
            kh, vh = k[b, h // (Hq // Hkv)].double(), v[b, h // (Hq // Hkv)].double()
            for r0 in range(0, Nq, step):
                s = q[b, h, r0:r0 + step].double() @ kh.T / math.sqrt(D)
                if causal:
                    rows = torch.arange(r0, r0 + s.shape[0], device=q.device) + (Nk - Nq)
                    s.masked_fill_(cols[None, :] > rows[:, None], float("-inf"))
                z = torch.logsumexp(s, 1)
                lse[b, h, r0:r0 + step] = z
                out[b, h, r0:r0 + step] = torch.exp_(s.sub_(z[:, None])) @ vh
    return out, lse


def exact(case, seed):
    """The outputs of ``run`` in 64 bits, in plain torch; None where that would take long."""
    c = case
    if c["B"] * c["Hq"] * c["Nq"] * c["Nk"] > 2e10:
        return None
    s = prepare(c, seed)
    if c["op"] == "module":
        m, x = s["m"], s["x"].double()
        lin = lambda layer, y: y @ layer.weight.double().T + layer.bias.double()  # noqa: E731
        B, N, d = x.shape
        q = lin(m.w_q, x).view(B, N, c["Hq"], c["D"]).transpose(1, 2)
        kv = lin(m.kv, x).view(B, N, 2, c["Hkv"], c["D"])
        o, _ = _attention64(q, kv[:, :, 0].transpose(1, 2), kv[:, :, 1].transpose(1, 2), True)
        return lin(m.w_o, o.transpose(1, 2).reshape(B, N, d))
    q, k, v = (t if c["layout"] == "bhnd" else t.transpose(1, 2) for t in (s["q"], s["k"], s["v"]))
    if c["op"] == "int8":
        mean = k.double().mean(2, keepdim=True).float()
        q, k = _quantised(q), _quantised(k.float() - mean)
    if c["op"] == "shard":
        G = c["Hq"] // c["Hkv"]
        out = torch.zeros(q.shape, dtype=torch.float64, device=q.device)
        for b, hk in parallel.shard_units(c["B"], c["Hkv"], c["world"], 0):
            qs = slice(hk * G, (hk + 1) * G)
            out[b:b + 1, qs] = _attention64(q[b:b + 1, qs], k[b:b + 1, hk:hk + 1], v[b:b + 1, hk:hk + 1], c["causal"])[0]
        return out
    o, lse = _attention64(q, k, v, c["causal"])
    if c["layout"] == "bnhd":
        o = o.transpose(1, 2)
    return (o, lse) if c["lse"] else o
