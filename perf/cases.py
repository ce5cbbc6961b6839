"""The attention work a user of this package has it do: what is timed, on which inputs, what one
pass cannot do without, and how far two correct implementations may differ.

A case is a dict of plain values.  ``op`` names the path:

* ``attend``    attention over operands that are quantised already (tiled or linear scales);
* ``prefill``   bf16 q, k, v in hand: quantise, then attend (a layer of a prompt pass);
* ``quantize``  the quantiser alone, on one layer's q, k, v;
* ``cache``     a few query tokens, or a chunk of a prompt, against a KV cache: contiguous or
                paged, every sequence with a length of its own;
* ``varlen``    a packed batch of sequences of unequal lengths;
* ``host``      operands in pinned host memory, result back in pinned host memory.

Sizes are those of the benchmark configurations, the tests and the sweep of this repository.
"""
import math
import random

import numpy as np
import torch

import flash_attention_b200 as fa


def listed():
    return [
        # one token of one sequence, scales as a plain quantiser writes them: latency is everything
        {"name": "decode_one", "op": "cache", "B": 1, "Sq": 1, "Sk": 777, "Hq": 32, "Hkv": 8, "paged": False,
         "ragged": False, "layout": "linear"},
        # one decode step of a serving batch: paged cache, every sequence with its own length
        {"name": "decode_paged", "op": "cache", "B": 16, "Sq": 1, "Sk": 8192, "Hq": 32, "Hkv": 8, "paged": True,
         "ragged": True, "layout": "tiled"},
        # a chunk of a long prompt against what the cache holds so far
        {"name": "chunk_long", "op": "cache", "B": 1, "Sq": 128, "Sk": 16384, "Hq": 32, "Hkv": 8, "paged": False,
         "ragged": False, "layout": "tiled"},
        # a short prompt of an odd length, from bf16 activations to the output
        {"name": "prefill_short", "op": "prefill", "B": 1, "S": 333, "Hq": 32, "Hkv": 8, "D": 128, "causal": True},
        # the non-causal benchmark configuration
        {"name": "dense_noncausal", "op": "attend", "B": 4, "Sq": 4096, "Sk": 4096, "Hq": 32, "Hkv": 32, "D": 128,
         "causal": False, "window": -1, "sink": False, "outliers": False, "layout": "tiled", "lse": True},
        # the headline benchmark configuration
        {"name": "dense_causal_gqa", "op": "attend", "B": 4, "Sq": 8192, "Sk": 8192, "Hq": 32, "Hkv": 8, "D": 128,
         "causal": True, "window": -1, "sink": False, "outliers": False, "layout": "tiled", "lse": True},
        # the long-context benchmark configuration: the largest call
        {"name": "dense_long_context", "op": "attend", "B": 1, "Sq": 32768, "Sk": 32768, "Hq": 64, "Hkv": 8, "D": 128,
         "causal": True, "window": -1, "sink": False, "outliers": True, "layout": "tiled", "lse": False},
        # a sliding-window layer with sinks, head dim 64
        {"name": "window_sink_d64", "op": "attend", "B": 2, "Sq": 4096, "Sk": 4096, "Hq": 64, "Hkv": 8, "D": 64,
         "causal": True, "window": 127, "sink": True, "outliers": False, "layout": "tiled", "lse": False},
        # a point of the shape sweep with the wide head dim, linear scales
        {"name": "dense_d192", "op": "attend", "B": 8, "Sq": 2048, "Sk": 2048, "Hq": 16, "Hkv": 16, "D": 192,
         "causal": True, "window": -1, "sink": False, "outliers": False, "layout": "linear", "lse": True},
        # a packed batch of prompts of very different lengths
        {"name": "varlen_packed", "op": "varlen", "seqs": 24, "longest": 2048, "Hq": 32, "Hkv": 8, "D": 128,
         "causal": True},
        # the quantiser on the q, k, v of the headline configuration
        {"name": "quantize_layer", "op": "quantize", "B": 4, "S": 8192, "Hq": 32, "Hkv": 8, "D": 128},
        # operands that live in host memory
        {"name": "host_buffers", "op": "host", "B": 2, "S": 4096, "Hq": 32, "Hkv": 8, "D": 128, "causal": True},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["cache", "cache", "cache", "attend", "attend", "attend", "prefill", "quantize", "varlen", "host"])
    Hq, Hkv = rng.choice([(32, 8), (32, 8), (64, 8), (16, 16), (32, 32), (8, 1)])
    D = rng.choice([128, 128, 128, 64, 192])
    if op == "cache":
        Sk = _log(rng, 128, 65536)
        B = _log(rng, 1, max(1, min(64, 524288 // Sk)))
        paged = rng.random() < 0.5
        Sq = rng.choice([1, 1, 1, 1, 2, 4, _log(rng, 33, 512)])
        if Hq // Hkv * Sq <= 32 and Sq > 1 and rng.random() < 0.5:
            Sq = 1
        Sq = min(Sq, Sk)
        if paged:
            Sk = (Sk + 127) // 128 * 128
        return {"op": "cache", "B": B, "Sq": Sq, "Sk": Sk, "Hq": Hq, "Hkv": Hkv, "paged": paged,
                "ragged": paged or rng.random() < 0.3, "layout": "tiled" if paged else rng.choice(["tiled", "linear"])}
    if op == "varlen":
        return {"op": "varlen", "seqs": _log(rng, 2, 128), "longest": _log(rng, 128, 4096), "Hq": Hq, "Hkv": Hkv, "D": D,
                "causal": rng.random() < 0.8}
    if op in ("quantize", "prefill", "host"):
        S = _log(rng, 64, 8192)
        B = _log(rng, 1, max(1, min(8, 16384 // S)))
        c = {"op": op, "B": B, "S": S, "Hq": Hq, "Hkv": Hkv, "D": 128 if op == "host" else D}
        if op != "quantize":
            c["causal"] = op == "prefill" or rng.random() < 0.7
        return c
    S = _log(rng, 128, 32768)
    while True:
        B = _log(rng, 1, 16)
        window = rng.choice([-1, -1, -1, 127, 1023])
        causal = window >= 0 or rng.random() < 0.6
        c = {"op": "attend", "B": B, "Sq": S, "Sk": S, "Hq": Hq, "Hkv": Hkv, "D": D, "causal": causal,
             "window": window, "sink": window >= 0 and rng.random() < 0.5, "outliers": rng.random() < 0.15,
             "layout": rng.choice(["tiled", "tiled", "linear"]), "lse": rng.random() < 0.5}
        if B * S * Hq <= 64 * 32768 and _pairs(c) * Hq <= 64 * 32768 * 32769 // 2:
            return c
        S = max(128, S // 2 + rng.randrange(64))


# ---- what a case consists of ---------------------------------------------------------------------

def _dv(D):
    return 128 if D == 192 else D


def _spread(n, longest):
    """n lengths up to `longest`, spread over the logarithm; the longest among them.  The same for
    every seed (a pass then has the same work); only their order in the batch changes with it."""
    r = random.Random(n * 1000003 + longest)
    lens = [_log(r, max(1, longest // 64), longest) for _ in range(n)]
    lens[0] = longest
    return lens


def _lengths(case):
    """(query length, key length) of every sequence of the batch."""
    op = case["op"]
    if op == "varlen":
        return [(s, s) for s in _spread(case["seqs"], case["longest"])]
    if op == "cache":
        keys = _spread(case["B"], case["Sk"]) if case["ragged"] else [case["Sk"]] * case["B"]
        return [(case["Sq"], max(n, case["Sq"])) for n in keys]
    if op == "attend":
        return [(case["Sq"], case["Sk"])] * case["B"]
    return [(case["S"], case["S"])] * case["B"]


def _pairs(case):
    """Visible (query, key) pairs of one query head, over the batch."""
    total, window = 0, case.get("window", -1)
    causal = case.get("causal", case["op"] == "cache")
    for (sq, sk), n in {p: _lengths(case).count(p) for p in set(_lengths(case))}.items():
        if not causal:
            total += n * sq * sk
            continue
        seen = np.arange(sk - sq + 1, sk + 1, dtype=np.int64)
        if window >= 0:
            seen = np.minimum(seen, window + 1)
        total += n * int(seen.sum())
    return total


def work(case):
    """Bytes: every operand (values and scales, the visible keys) once, every result once.  FLOPs:
    the two products over the visible pairs."""
    D, Hq, Hkv = case.get("D", 128), case["Hq"], case["Hkv"]
    Dv = _dv(D)
    nq = sum(sq for sq, _ in _lengths(case))
    nk = sum(sk for _, sk in _lengths(case))
    e = 0.5 + 1.0 / 16                                       # packed bytes per element, scales included
    elements = nq * Hq * D + nk * Hkv * D + nk * Hkv * Dv
    if case["op"] == "quantize":
        return {"bytes": elements * (2 + e), "flops": 4.0 * elements}    # maximum, scale, round, compare
    out = nq * Hq * (2 * Dv + (4 if case.get("lse", case["op"] in ("varlen", "host")) else 0))
    return {"bytes": elements * (2 if case["op"] == "prefill" else e) + out,
            "flops": 2.0 * (D + Dv) * Hq * _pairs(case)}


def tolerance(case):
    """The quantiser's bytes and scales are defined to the bit.  Attention: bf16 results of fp32
    sums; a weight next to a rounding boundary of its 4-bit format may fall to the other side, which
    a row with few keys shows most."""
    return "exact" if case["op"] == "quantize" else {"rel": 0.01, "max": 0.5}


# ---- inputs --------------------------------------------------------------------------------------

def _activations(g, B, Sq, Sk, Hq, Hkv, D, outliers=False):
    """bf16 q, k, v in the (batch, seq, heads, dim) layout; `outliers`: 1 % of the channels of q and k x20."""
    q, k, v = (torch.randn(B, S, H, d, generator=g, device="cuda", dtype=torch.bfloat16)
               for S, H, d in ((Sq, Hq, D), (Sk, Hkv, D), (Sk, Hkv, _dv(D))))
    if outliers:
        for t in (q, k):
            at = torch.randperm(D, generator=g, device="cuda")[:max(1, round(0.01 * D))]
            t[..., at] *= 20.0
    return q, k, v


def _as_given(t, layout):
    """What the program holds of a quantised operand: its bytes, its scales in the one layout, its scale."""
    return t.data, (t.sf if layout == "linear" else t.tiled_sf()), t.scale


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    op, Hq, Hkv, D = case["op"], case["Hq"], case["Hkv"], case.get("D", 128)
    st = {"case": case}
    if op in ("quantize", "prefill"):
        st["qkv"] = _activations(g, case["B"], case["S"], case["S"], Hq, Hkv, D)
    elif op == "attend":
        qkv = fa.quantize_qkv_fused(*_activations(g, case["B"], case["Sq"], case["Sk"], Hq, Hkv, D, case["outliers"]))
        if case["layout"] == "tiled":
            st["qkv"] = tuple(fa.NVFP4Tensor(t.data, t.tiled_sf(), t.scale, True, t.is_v) for t in qkv)
        else:
            st["qkv"] = tuple(fa.NVFP4Tensor(t.data, t.sf, t.scale, False, t.is_v) for t in qkv)
        st["sink"] = torch.randn(Hq, generator=g, device="cuda") if case["sink"] else None
    elif op == "cache":
        B, Sk = case["B"], case["Sk"]
        lens = [n for _, n in _lengths(case)]
        random.Random(seed).shuffle(lens)
        pages = -(-Sk // 128)
        # the cache: B rows of Sk slots, or a pool of pages of 128 slots in an order of its own
        rows, slots = (B * pages, 128) if case["paged"] else (B, Sk)
        q, k, v = _activations(g, 1, B * case["Sq"], rows * slots, Hq, Hkv, 128)
        Q, K, V = fa.quantize_qkv_fused(q.view(B, case["Sq"], Hq, 128), k.view(rows, slots, Hkv, 128),
                                        v.view(rows, slots, Hkv, 128))
        st["q"], st["k"], st["v"] = (_as_given(t, case["layout"]) for t in (Q, K, V))
        st["used"] = torch.tensor(lens, dtype=torch.int32, device="cuda") if case["ragged"] else None
        st["table"] = None
        if case["paged"]:
            st["table"] = torch.randperm(rows, generator=g, device="cuda").to(torch.int32).view(B, pages)
    elif op == "varlen":
        lens = [n for n, _ in _lengths(case)]
        random.Random(seed).shuffle(lens)
        cu = np.concatenate([[0], np.cumsum(lens)])
        st["cu"] = torch.tensor(cu, dtype=torch.int32, device="cuda")
        st["longest"] = max(lens)
        q, k, v = _activations(g, 1, int(cu[-1]), int(cu[-1]), Hq, Hkv, D)
        Q, K, V, st["cu_v"] = fa.quantize_varlen_qkv(q[0], k[0], v[0], st["cu"],
                                                     total_v=sum(-(-n // 32) * 32 for n in lens))
        st["q"], st["k"], st["v"] = ((t.data[0], t.sf[0], t.scale) for t in (Q, K, V))
    elif op == "host":
        B, S = case["B"], case["S"]
        Q, K, V = fa.quantize_qkv_fused(*_activations(g, B, S, S, Hq, Hkv, D))
        st["operands"] = [x.cpu().pin_memory() for x in (Q.data, K.data, V.data, Q.sf, K.sf, V.sf)]
        st["scales"] = [Q.scale, K.scale, V.scale]
        st["pipe"] = fa.HostPipeline(B, S, S, Hq, Hkv, D, _dv(D))
        st["out"] = torch.empty(B, S, Hq, _dv(D), dtype=torch.bfloat16).pin_memory()
        st["lse"] = torch.empty(B, Hq, S, dtype=torch.float32).pin_memory()
    else:
        raise ValueError(op)
    return st


def run(st):
    case = st["case"]
    op = case["op"]
    if op == "attend":
        window = (None, None) if case["window"] < 0 else (case["window"], 0)
        return fa.flash_attn_func(*st["qkv"], causal=case["causal"], window_size=window, learnable_sink=st["sink"],
                                  return_lse=case["lse"])
    if op == "prefill":
        return fa.flash_attn_func(*fa.quantize_qkv_fused(*st["qkv"]), causal=case["causal"])[0]
    if op == "quantize":
        return [(t.data, t.sf, t.sf_tiled, t.scale) for t in fa.quantize_qkv_fused(*st["qkv"])]
    if op == "cache":
        (q, q_sf, q_g), (k, k_sf, k_g), (v, v_sf, v_g) = st["q"], st["k"], st["v"]
        return fa.flash_attn_fp4_func(q, k, v, q_sf, k_sf, v_sf, q_g, k_g, v_g, causal=True, sf_layout=case["layout"],
                                      num_splits=0, seqused_k=st["used"], page_table=st["table"])[0]
    if op == "varlen":
        (q, q_sf, q_g), (k, k_sf, k_g), (v, v_sf, v_g) = st["q"], st["k"], st["v"]
        return fa.flash_attn_varlen_fp4_func(q, k, v, q_sf, k_sf, v_sf, q_g, k_g, v_g, st["cu"], st["cu"],
                                             cu_seqlens_v=st["cu_v"], max_seqlen_q=st["longest"],
                                             max_seqlen_k=st["longest"], causal=case["causal"], return_lse=True)
    # the caller reads the result on the host, so it waits for it
    st["pipe"].run(*st["operands"], *st["scales"], st["out"], st["lse"], causal=case["causal"])
    st["pipe"].wait()
    return st["out"], st["lse"]
