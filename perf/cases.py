"""Attention workloads that measure this library: what a training step, a serving step and the feature-major
boundary ask of it, through the Python entry points of ``sentinel_b200``.

Every case is a dict of plain values.  ``kind`` names the path:

* ``train``   attention_forward + attention_backward on token-major ``[B, H, S, D]`` tensors (bf16 or fp32), causal,
              optionally with a sliding window and global tokens or with bit-reproducible dQ;
* ``matrix``  CudaFlashAttention.forwardMultiHead + backwardMultiHead on fp32 feature-major matrices, exact or (``reduced``)
              with bf16 tensor-core operands: the call a Sentinel build makes;
* ``cached``  attention_cached_forward: one or more new tokens against a KV cache (decode, continued prefill);
* ``rope``    the boundary of one layer: pack Q, K (rotated), V, dO into bf16 heads, unpack O, dQ, dK (inverse rotation), dV.
"""
import math

import torch

import sentinel_b200 as sb
from sentinel_b200.flash_attention import CudaFlashAttention

DETERMINISTIC = 4   # SNTL_FLAG_DETERMINISTIC of include/sntl_attn.h


def train(name, B, Hq, Hkv, S, D, dtype="bf16", window=0, global_tokens=0, flags=0):
    return dict(name=name, kind="train", B=B, Hq=Hq, Hkv=Hkv, S=S, D=D, dtype=dtype, window=window,
                global_tokens=global_tokens, flags=flags)


def matrix(name, packs, Hq, Hkv, S, D, reduced, column_start=0):
    return dict(name=name, kind="matrix", B=packs, Hq=Hq, Hkv=Hkv, S=S, D=D, reduced=reduced, column_start=column_start)


def cached(name, B, Hq, Hkv, T, L, capacity, D, dtype="bf16"):
    return dict(name=name, kind="cached", B=B, Hq=Hq, Hkv=Hkv, T=T, L=L, capacity=capacity, D=D, dtype=dtype)


def rope(name, B, Hq, Hkv, S, D):
    return dict(name=name, kind="rope", B=B, Hq=Hq, Hkv=Hkv, S=S, D=D)


def listed():
    return [
        # the toy model that the repository's parity bar is quoted on: nothing but launches and latency
        train("toy_f32", 4, 4, 4, 64, 16, dtype="f32"),
        # a 12-layer, 768-wide model trained in fp32 matrices: 8 packed sequences of 512 tokens per microstep, exact kernels
        matrix("matrix_f32_768", 8, 12, 12, 512, 64, reduced=False),
        # a 2048-wide model with 32 heads, 2 packs of 1024 tokens, bf16 operands allowed: staging copies around the kernels
        matrix("matrix_bf16_2048", 2, 32, 32, 1024, 64, reduced=True),
        # training steps of the three bf16 model shapes the benchmark names: small multi-head, 1B grouped-query, 7B-class
        train("gpt2_small", 8, 12, 12, 1024, 64),
        train("llama1b_gqa", 4, 32, 8, 4096, 64),
        train("gqa7b_d128", 2, 28, 4, 8192, 128),
        # the 7B-class layer with a sliding window and always-visible first tokens
        train("gqa7b_window", 2, 28, 4, 8192, 128, window=1024, global_tokens=64),
        # fine-tuning on documents of an odd length, with bit-reproducible input gradients
        train("ragged_deterministic", 3, 16, 4, 1237, 128, flags=DETERMINISTIC),
        # a prompt continued from a cache: 512 new tokens behind 3587 cached ones
        cached("chunked_prefill", 1, 28, 4, 512, 4099, 8192, 128),
        # serving: one new token for each of 64 sequences
        cached("decode_batch64", 64, 28, 4, 1, 8192, 8192, 128),
        # one fp32 sequence being generated by the 768-wide model
        cached("decode_f32_single", 1, 12, 12, 1, 777, 1024, 64, dtype="f32"),
        # the boundary conversions of one 7B-class layer, forward and backward
        rope("rope_boundary_7b", 2, 28, 4, 8192, 128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _heads(rng, kv=(1, 2, 4, 8), groups=(1, 2, 4, 7)):
    hkv = rng.choice(kv)
    return hkv * rng.choice(groups), hkv


# Most (sequence, KV head) units of a drawn bf16 call at head_dim 64: with more of them the backward had a race between its
# warpgroups when this file was written, and outputs that are wrong now and then are nothing to compare with.
UNITS_D64 = 64


def draw(rng):
    kind = rng.choice(["train", "train", "train", "train_f32", "matrix", "matrix", "cached", "cached", "cached_f32", "rope"])
    if kind == "train":
        D = rng.choice([64, 128])
        Hq, Hkv = rng.choice([_heads(rng), (12, 12), (16, 16)])
        S = _log(rng, 64, 8192)
        # at most the largest listed step's products and activations
        most = max(1, int(min(3.3e12 / (7.0 * Hq * S * S * D), 4.0e8 / (Hq * S * D * 2))))
        if D == 64:
            most = min(most, UNITS_D64 // Hkv)
        c = train("", min(most, _log(rng, 1, 16)), Hq, Hkv, S, D)
        style = rng.random()
        if style < 0.25:
            c.update(window=_log(rng, 64, 4096), global_tokens=rng.choice([0, 4, 64, 130]))
        elif style < 0.4:
            c.update(flags=DETERMINISTIC)
    elif kind == "train_f32":
        Hq, Hkv = _heads(rng, groups=(1, 2, 3))
        c = train("", _log(rng, 1, 8), Hq, Hkv, _log(rng, 16, 512), rng.choice([16, 32, 64, 80, 96, 128]), dtype="f32")
        while c["B"] > 1 and 7.0 * c["B"] * Hq * c["S"] ** 2 * c["D"] > 1.2e10:
            c["B"] -= 1
    elif kind == "matrix":
        reduced = rng.random() < 0.5
        Hq, Hkv = rng.choice([(4, 4), (8, 8), (12, 12), (8, 2), (12, 4), (16, 4)] + ([(32, 8), (48, 48), (48, 16)] if reduced else []))
        # sequences are bucketed to 32 tokens; a single unpacked one may have any length
        S, packs = 32 * _log(rng, 1, 16), _log(rng, 1, 8)
        if rng.random() < 0.25:
            S, packs = _log(rng, 33, 700), 1
        D = rng.choice([64, 64, 128]) if reduced else rng.choice([32, 64])
        if reduced and D == 64:
            packs = min(packs, UNITS_D64 // Hkv)
        c = matrix("", packs, Hq, Hkv, S, D, reduced=reduced, column_start=rng.choice([0, 0, 32]))
    elif kind == "cached":
        D = rng.choice([64, 128])
        Hq, Hkv = rng.choice([(28, 4), (32, 8), (8, 2), (12, 12)])
        T = 1 if rng.random() < 0.7 else _log(rng, 2, 1024)
        L = max(T, _log(rng, 128, 16384))
        most = max(1, int(1.0e9 / (4.0 * Hkv * L * D)))
        B = min(most, 64 if T == 1 else 4, _log(rng, 1, 64))
        c = cached("", B, Hq, Hkv, T, L, L if rng.random() < 0.5 else L + _log(rng, 1, 1024), D)
    elif kind == "cached_f32":
        Hq, Hkv = rng.choice([(4, 4), (8, 8), (12, 12), (12, 4)])
        T = 1 if rng.random() < 0.7 else _log(rng, 2, 32)
        L = max(T, _log(rng, 32, 2048))
        c = cached("", _log(rng, 1, 4), Hq, Hkv, T, L, L + _log(rng, 1, 512), rng.choice([32, 64, 128]), dtype="f32")
    else:
        D = rng.choice([64, 128])
        Hq, Hkv = rng.choice([(28, 4), (32, 8), (12, 12), (8, 2)])
        S = _log(rng, 64, 8192)
        c = rope("", max(1, min(_log(rng, 1, 8), int(2 * 28 * 8192 * 128 / (Hq * S * D)))), Hq, Hkv, S, D)
    del c["name"]
    return c


def _randn(g, *shape, std=1.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=g, device="cuda") * std).to(dtype)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, Hq, Hkv, D = case["B"], case["Hq"], case["Hkv"], case["D"]
    st = {"case": case}
    if case["kind"] == "train":
        dt, S = (torch.bfloat16, case["S"]) if case["dtype"] == "bf16" else (torch.float32, case["S"])
        # post-RoPE projections of a trained layer; gradients are small.  fp32: the unit normals of the toy model
        qk, do = (0.5, 1e-2) if case["dtype"] == "bf16" else (1.0, 1.0)
        st.update(q=_randn(g, B, Hq, S, D, std=qk, dtype=dt), k=_randn(g, B, Hkv, S, D, std=qk, dtype=dt),
                  v=_randn(g, B, Hkv, S, D, dtype=dt), do=_randn(g, B, Hq, S, D, std=do, dtype=dt))
    elif case["kind"] == "matrix":
        S, col = case["S"], case["column_start"]
        C = col + B * S
        st.update(q=_randn(g, Hq * D, C, std=0.5), k=_randn(g, Hkv * D, C, std=0.5), v=_randn(g, Hkv * D, C), do=_randn(g, Hq * D, C, std=1e-2))
        # the layer's own persistent result matrices
        for n, rows in (("out", Hq * D), ("lse", Hq), ("dq", Hq * D), ("dk", Hkv * D), ("dv", Hkv * D)):
            st[n] = torch.zeros(rows, C, device="cuda")
    elif case["kind"] == "cached":
        dt = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
        st.update(q=_randn(g, B, Hq, case["T"], D, std=0.5, dtype=dt), k=_randn(g, B, Hkv, case["capacity"], D, std=0.5, dtype=dt),
                  v=_randn(g, B, Hkv, case["capacity"], D, dtype=dt))
    else:
        S = case["S"]
        for n, H in (("q", Hq), ("k", Hkv), ("v", Hkv), ("do", Hq)):
            st[n] = _randn(g, H * D, B * S, std=0.5)
        for n, H in (("o", Hq), ("dq", Hq), ("dk", Hkv), ("dv", Hkv)):
            st[n] = _randn(g, B, H, S, D, std=0.5, dtype=torch.bfloat16)
            st[n + "_matrix"] = torch.zeros(H * D, B * S, device="cuda")
        angle = torch.arange(S, device="cuda", dtype=torch.float32)[:, None] * \
            torch.pow(torch.tensor(1e6, device="cuda"), -2.0 * torch.arange(D // 2, device="cuda", dtype=torch.float32) / D)[None, :]
        st.update(cos=torch.cos(angle).contiguous(), sin=torch.sin(angle).contiguous())
    return st


def run(st):
    c = st["case"]
    if c["kind"] == "train":
        o, lse = sb.attention_forward(st["q"], st["k"], st["v"], flags=c["flags"], window=c["window"], global_tokens=c["global_tokens"])
        dq, dk, dv = sb.attention_backward(st["q"], st["k"], st["v"], o, lse, st["do"], flags=c["flags"], window=c["window"],
                                           global_tokens=c["global_tokens"])
        return o, lse, dq, dk, dv
    if c["kind"] == "matrix":
        CudaFlashAttention.allow_reduced_precision = c["reduced"]
        shape = (c["Hq"], c["D"], c["D"] ** -0.5, True, c["column_start"], c["S"], c["B"])
        CudaFlashAttention.forwardMultiHead(st["q"], st["k"], st["v"], st["out"], st["lse"], *shape)
        CudaFlashAttention.backwardMultiHead(st["q"], st["k"], st["v"], st["out"], st["lse"], st["do"], st["dq"], st["dk"], st["dv"],
                                             None, *shape)
        return st["out"], st["lse"], st["dq"], st["dk"], st["dv"]
    if c["kind"] == "cached":
        return sb.attention_cached_forward(st["q"], st["k"], st["v"], c["L"])
    B, Hq, Hkv, S, D = c["B"], c["Hq"], c["Hkv"], c["S"], c["D"]
    angles = dict(cos_table=st["cos"], sin_table=st["sin"])
    q = sb.pack_heads(st["q"], B, Hq, S, D, **angles)
    k = sb.pack_heads(st["k"], B, Hkv, S, D, **angles)
    v = sb.pack_heads(st["v"], B, Hkv, S, D)
    o = sb.unpack_heads(st["o"], st["o_matrix"])
    do = sb.pack_heads(st["do"], B, Hq, S, D)
    dq = sb.unpack_heads(st["dq"], st["dq_matrix"], inverse=True, **angles)
    dk = sb.unpack_heads(st["dk"], st["dk_matrix"], inverse=True, **angles)
    dv = sb.unpack_heads(st["dv"], st["dv_matrix"])
    return q, k, v, o, do, dq, dk, dv


def _visible_pairs(S, window, global_tokens):
    """(query, key) pairs of one head that the causal mask, the window and the global tokens leave visible."""
    if window <= 0 or window >= S:
        return S * (S + 1) // 2
    pairs = window * (window + 1) // 2 + (S - window) * window
    # query i also sees the global keys below its window, min(global_tokens, i - window + 1) of them
    beyond = S - window
    g = min(global_tokens, beyond)
    return pairs + g * (g + 1) // 2 + (beyond - g) * g


def work(case):
    B, Hq, Hkv, D = case["B"], case["Hq"], case["Hkv"], case["D"]
    if case["kind"] in ("train", "matrix"):
        S = case["S"]
        size = 2 if case["kind"] == "train" and case["dtype"] == "bf16" else 4
        pairs = _visible_pairs(S, case.get("window", 0), case.get("global_tokens", 0))
        # reads Q, dO, K, V; writes O, dQ, dK, dV and the fp32 log-sum-exp; 2 + 5 products
        return {"bytes": size * B * S * D * (4 * Hq + 4 * Hkv) + 4 * B * Hq * S, "flops": 14.0 * B * Hq * pairs * D}
    if case["kind"] == "cached":
        T, L = case["T"], case["L"]
        size = 2 if case["dtype"] == "bf16" else 4
        pairs = T * (L - T) + T * (T + 1) // 2
        return {"bytes": size * B * D * (2 * Hq * T + 2 * Hkv * L) + 4 * B * Hq * T, "flops": 4.0 * B * Hq * pairs * D}
    S = case["S"]
    return {"bytes": 6 * B * S * D * (4 * Hq + 4 * Hkv) + 4 * S * D, "flops": 0.0}


def tolerance(case):
    if case["kind"] == "rope":
        return "exact"   # products and sums rounded one by one, then to bf16: a bit pattern
    if case.get("dtype") == "f32" or case.get("reduced") is False:
        return {"rel": 1e-5}
    return {"rel": 1e-2}   # bf16 operands, P and dS rounded to bf16 between the products
