"""The work a user of racetrack_b200 has it do, as cases to time: what each one is, its inputs, one
pass through the public entry points, the bytes and operations that pass cannot do without, and how
far two correct evaluations of it may lie apart.

Sizes are those of the DeepSeek-V3.2 block this package serves (hidden 7168, 128 heads, MLA ranks
1536 / 512, 256 experts x 2048 with top-8, dense FFN 18432, indexer 64 x 128 with top-2048) and of
the token counts bench.py, kernel_bench.py and the tests run it at.
"""
from __future__ import annotations

import math

import torch

from racetrack_b200 import decode, indexer, layer, moe, ops

HIDDEN, Q_LORA, KV_LORA, NOPE, ROPE, V_DIM, HEADS = 7168, 1536, 512, 128, 64, 128, 128
EXPERTS, TOPK, INTER, DENSE_INTER = 256, 8, 2048, 18432
INDEX_HEADS, INDEX_DIM, INDEX_TOPK = 64, 128, 2048
QKV_A, QK = Q_LORA + KV_LORA + ROPE, NOPE + ROPE
EPS = 1.0e-6

BF16, F32 = torch.bfloat16, torch.float32


def listed() -> list[dict]:
    return [
        # the partition's element-wise MLA prologue (residual add + RMSNorm, q_a / kv_a RMSNorm with
        # the k_pe rotation, q_pe rotation): a small batch, where launches count, and a long prompt
        {"name": "prologue_128", "kind": "prologue", "tokens": 128},
        {"name": "prologue_5003", "kind": "prologue", "tokens": 5003},
        # SwiGLU of the dense FFN's gate_up with both activation quantisers behind it
        {"name": "swiglu_quant_4096", "kind": "swiglu_quant", "tokens": 4096},
        # the sparse-attention indexer on the second half of a 4096-token prompt
        {"name": "indexer_2048", "kind": "indexer", "tokens": 2048, "start": 2048},
        # a routed MoE layer with its gate and shared expert: a single token, and a prefill chunk
        {"name": "moe_1", "kind": "moe", "tokens": 1},
        {"name": "moe_4096", "kind": "moe", "tokens": 4096},
        # one layer of a decode step over caches of some thousand positions: a single sequence, a
        # few sequences with a short odd context (every position attended to) and the long
        # projections in FP8, a full batch
        {"name": "decode_1", "kind": "decode", "batch": 1, "context": 4096, "proj": "bf16"},
        {"name": "decode_13", "kind": "decode", "batch": 13, "context": 1537, "proj": "mixed"},
        {"name": "decode_64", "kind": "decode", "batch": 64, "context": 4096, "proj": "bf16"},
        # one layer of a prefill: a short ragged prompt, the dense layers of the model with FP8
        # projections, and the largest batch of tokens (bench.py's own step, one layer of it)
        {"name": "prefill_777", "kind": "prefill", "tokens": 777, "ffn": "moe", "proj": "bf16"},
        {"name": "dense_2048", "kind": "prefill", "tokens": 2048, "ffn": "dense", "proj": "fp8"},
        {"name": "prefill_8192", "kind": "prefill", "tokens": 8192, "ffn": "moe", "proj": "mixed"},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["prologue", "swiglu_quant", "indexer", "moe", "moe", "decode", "decode", "prefill", "prefill"])
    if kind == "prologue":
        return {"kind": kind, "tokens": _log_int(rng, 1, 8192)}
    if kind == "swiglu_quant":
        return {"kind": kind, "tokens": _log_int(rng, 1, 4096)}
    if kind == "indexer":
        return {"kind": kind, "tokens": _log_int(rng, 129, 2048), "start": rng.randrange(0, 4096)}
    if kind == "moe":
        return {"kind": kind, "tokens": _log_int(rng, 1, 4096)}
    if kind == "decode":
        return {"kind": kind, "batch": _log_int(rng, 1, 64), "context": _log_int(rng, 64, 4096),
                "proj": rng.choice(["bf16", "mixed", "fp8"])}
    return {"kind": kind, "tokens": _log_int(rng, 129, 8192), "ffn": rng.choice(["moe", "dense"]),
            "proj": rng.choice(["bf16", "mixed", "fp8"])}


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------

def _shape(seed: int) -> layer.LayerShape:
    """The layer's dimensions with weights of this seed (each weight has a seed of its own behind it)."""
    return layer.DSV32.scaled(seed=38595 + 1_000_003 * (seed % 2_000_003))


def _normal(gen, *size, mean: float = 0.0, std: float = 1.0, dtype=BF16):
    return torch.empty(*size, device="cuda", dtype=F32).normal_(mean, std, generator=gen).to(dtype)


def _freqs(positions: int):
    return decode.rope_table(ROPE, positions, 10000.0, "cuda")


def _layer_rows(s: dict, gen, rows: int) -> None:
    """The inputs of a layer's two halves: normalised rows and the residual stream at each. The feed-
    forward half gets rows of its own instead of the attention half's result, because the NVFP4
    quantiser of the experts turns a last-bit difference of its input into a whole code: end to end,
    two correct evaluations of one layer lie 3 - 6 % apart, half by half a tenth of that."""
    for half in ("attn", "ffn"):
        s[half + "_in"], s[half + "_residual"] = _normal(gen, rows, HIDDEN), _normal(gen, rows, HIDDEN)


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = {"case": case}
    if kind == "prologue":
        t = case["tokens"]
        s["update"], s["residual"] = _normal(gen, t, HIDDEN), _normal(gen, t, HIDDEN)
        s["w_h"] = _normal(gen, HIDDEN, mean=1.0, std=0.02, dtype=F32)
        s["qkv"] = _normal(gen, t, QKV_A)
        s["w_q"] = _normal(gen, Q_LORA, mean=1.0, std=0.02, dtype=F32)
        s["w_kv"] = _normal(gen, KV_LORA, mean=1.0, std=0.02, dtype=F32)
        s["q_pe"] = _normal(gen, t, HEADS, ROPE)
        s["freqs"] = _freqs(t)
    elif kind == "swiglu_quant":
        s["gate_up"] = _normal(gen, case["tokens"], 2 * DENSE_INTER)
    elif kind == "indexer":
        t, end = case["tokens"], case["start"] + case["tokens"]
        s["weights"] = decode.make_indexer_weights(_shape(seed), "cuda")
        s["x"], s["qr"] = _normal(gen, t, HIDDEN), _normal(gen, t, Q_LORA)
        s["freqs"] = _freqs(end)
        codes, scales = ops.fused_act_quant(_normal(gen, end, INDEX_DIM))
        s["k_cache"], s["k_scale"] = codes, scales.view(end)
    elif kind == "moe":
        s["x"] = _normal(gen, case["tokens"], HIDDEN)
        s["gate"] = _normal(gen, EXPERTS, HIDDEN, std=0.02)
        s["bias"] = torch.empty(EXPERTS, device="cuda").uniform_(-0.1, 0.1, generator=gen)
        s["experts"] = layer.make_nvfp4_experts(_shape(seed), 0, 1, "cuda")
        s["shared_w13"] = _normal(gen, 2 * INTER, HIDDEN, std=0.02)
        s["shared_w2"] = _normal(gen, HIDDEN, INTER, std=0.02)
    elif kind == "decode":
        shape, b = _shape(seed), case["batch"]
        w = layer.make_weights(shape, 0, 1, "cuda", ffn="none")
        w["experts"] = layer.make_nvfp4_experts(shape, 0, 1, "cuda")
        # the caches hold the context before the new token, plus room for tokens to come
        caches = decode.DecodeCaches(shape, b, case["context"] + 64, "cuda", seed=seed % 997, fill=case["context"] - 1)
        s["layer"] = decode.DecodeLayer(shape, w, index_weights=decode.make_indexer_weights(shape, "cuda"),
                                        caches=caches, proj=case["proj"])
        _layer_rows(s, gen, b)
    elif kind == "prefill":
        shape, t = _shape(seed), case["tokens"]
        dense = case["ffn"] == "dense"
        w = layer.make_weights(shape, 0, 1, "cuda", ffn="dense" if dense else "none")
        if not dense:
            w["experts"] = layer.make_nvfp4_experts(shape, 0, 1, "cuda")
        s["layer"] = layer.RealisticLayer(shape, w, ffn=case["ffn"], proj=case["proj"])
        _layer_rows(s, gen, t)
        s["positions"] = torch.arange(t, device="cuda")
    else:
        raise ValueError(f"unknown kind {kind!r}")
    return s


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------

def run(s: dict):
    case = s["case"]
    kind = case["kind"]
    if kind == "prologue":
        normed, hidden = ops.fused_residual_norm(s["update"], s["residual"], s["w_h"], eps=EPS)
        qkv = s["qkv"]
        q_c, kv_c, k_pe = ops.fused_norm_rope_interleaved(
            qkv[:, :Q_LORA], s["w_q"], qkv[:, Q_LORA:Q_LORA + KV_LORA], s["w_kv"],
            qkv[:, Q_LORA + KV_LORA:], s["freqs"], eps=EPS)
        q_pe = ops.fused_rope(s["q_pe"], s["freqs"])
        return [normed, hidden, q_c, kv_c, k_pe, q_pe]
    if kind == "swiglu_quant":
        gate, up = s["gate_up"][:, :DENSE_INTER], s["gate_up"][:, DENSE_INTER:]
        c8, s8 = ops.fused_swiglu_quant(gate, up)
        c4, s4, g4 = ops.fused_swiglu_nvfp4_quant(gate, up)
        return [c8.view(torch.uint8), s8, c4, s4.view(torch.uint8), g4]
    if kind == "indexer":
        picked = indexer.indexer_forward(s["x"], s["qr"], s["weights"], s["k_cache"], s["k_scale"],
                                         case["start"], s["freqs"], INDEX_TOPK)
        # the model scatters the positions into a mask: they are a set, not a sequence
        mask = torch.zeros(case["tokens"], case["start"] + case["tokens"], dtype=torch.bool, device="cuda")
        mask.scatter_(1, picked.long(), True)
        return [mask, s["k_cache"].view(torch.uint8), s["k_scale"]]
    if kind == "moe":
        x = s["x"]
        gate_up = ops.linear_bf16(x, s["shared_w13"])
        shared = ops.linear_bf16(ops.fused_swiglu(gate_up[:, :INTER], gate_up[:, INTER:]), s["shared_w2"])
        return moe.fused_moe_forward(x, s["gate"], s["bias"], s["experts"], n_experts=EXPERTS, n_groups=8,
                                     topk_groups=4, topk=TOPK, route_scale=2.5, shared=shared)
    # one layer, as decode_stack / forward_stack of the layer string it together
    lay = s["layer"]
    if kind == "decode":
        attn = lay.decode_attention(s["attn_in"], case["context"] - 1)
    else:
        attn = lay.attention(s["attn_in"], s["positions"])
    attn_normed, attn_hidden = ops.fused_residual_norm(attn, s["attn_residual"], lay.ones_h, eps=EPS)
    ffn = lay.ffn_forward(s["ffn_in"])
    ffn_normed, ffn_hidden = ops.fused_residual_norm(ffn, s["ffn_residual"], lay.ones_h, eps=EPS)
    out = [attn_normed, attn_hidden, ffn, ffn_normed, ffn_hidden]
    # among more cached positions than the indexer keeps, near-ties decide which ones attention sees,
    # and the update alone (a mean over random values) follows them; the residual stream hardly does
    if kind != "decode" or case["context"] <= INDEX_TOPK:
        out.append(attn)
    if kind == "decode":
        c = lay.caches
        out += [c.kv, c.pe, c.index_k.view(torch.uint8), c.index_scale]
    return out


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------

def _weight_bytes(n: int, k: int, proj: str) -> float:
    fp8 = proj == "fp8" or (proj == "mixed" and k >= 4096)
    return n * k * (1 + 4 / 16384 if fp8 else 2)


def _experts(tokens: int) -> tuple[float, float]:
    """(bytes, flops) of the routed experts of `tokens` tokens: the NVFP4 weights of the experts that
    a uniform router touches, and every (token, expert) pair's two products."""
    touched = EXPERTS * (1.0 - (1.0 - TOPK / EXPERTS) ** tokens)
    return touched * 3 * INTER * HIDDEN * 9 / 16, 2.0 * tokens * TOPK * 3 * INTER * HIDDEN


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "prologue":
        t = case["tokens"]
        return {"bytes": t * (4 * HIDDEN + 2 * QKV_A + 2 * HEADS * ROPE) * 2 + t * ROPE * 4
                + (HIDDEN + Q_LORA + KV_LORA) * 4, "flops": t * (8 * HIDDEN + 5 * QKV_A + 6 * HEADS * ROPE)}
    if kind == "swiglu_quant":
        n = case["tokens"] * DENSE_INTER
        return {"bytes": n * 4 + n * (1 + 4 / 128) + n * (1 / 2 + 1 / 16), "flops": 12 * n}
    if kind == "indexer":
        t, start = case["tokens"], case["start"]
        end = start + t
        n_w = INDEX_HEADS * INDEX_DIM * Q_LORA * 2 + INDEX_DIM * HIDDEN * 2 + INDEX_HEADS * HIDDEN * 4
        pairs = t * start + t * (t + 1) // 2                 # (query, cached key) pairs under the mask
        proj = 2.0 * t * (INDEX_HEADS * INDEX_DIM * Q_LORA + (INDEX_DIM + INDEX_HEADS) * HIDDEN)
        # the mask in, the caches in and the new rows out
        return {"bytes": n_w + t * (HIDDEN + Q_LORA) * 2 + end * (INDEX_DIM + 4) + t * (INDEX_DIM + 4) + t * end,
                "flops": proj + 2.0 * pairs * INDEX_HEADS * INDEX_DIM}
    if kind == "moe":
        t = case["tokens"]
        eb, ef = _experts(t)
        dense = EXPERTS * HIDDEN + 3 * INTER * HIDDEN
        return {"bytes": eb + dense * 2 + 2 * t * HIDDEN * 2, "flops": ef + 2.0 * t * dense}
    if kind == "decode":
        b, ctx, proj = case["batch"], case["context"], case["proj"]
        eb, ef = _experts(b)
        kept = min(ctx, INDEX_TOPK)
        n_bf16 = (HEADS * (NOPE + V_DIM) * KV_LORA + EXPERTS * HIDDEN + INDEX_HEADS * INDEX_DIM * Q_LORA
                  + INDEX_DIM * HIDDEN)
        n_proj = QKV_A * HIDDEN + HEADS * QK * Q_LORA + HIDDEN * HEADS * V_DIM
        weights = (n_bf16 * 2 + INDEX_HEADS * HIDDEN * 4 + _weight_bytes(QKV_A, HIDDEN, proj)
                   + _weight_bytes(HEADS * QK, Q_LORA, proj) + _weight_bytes(HIDDEN, HEADS * V_DIM, proj))
        caches = b * ctx * (INDEX_DIM + 4) + b * kept * (KV_LORA + ROPE) * 2
        flops = (ef + 2.0 * b * (n_bf16 + n_proj + INDEX_HEADS * HIDDEN) + 2.0 * b * ctx * INDEX_HEADS * INDEX_DIM
                 + 2.0 * b * HEADS * kept * (2 * KV_LORA + ROPE))
        return {"bytes": eb + weights + caches + 10 * b * HIDDEN * 2, "flops": flops}
    t, proj = case["tokens"], case["proj"]
    n_proj = QKV_A * HIDDEN + HEADS * QK * Q_LORA + HEADS * (NOPE + V_DIM) * KV_LORA + HIDDEN * HEADS * V_DIM
    weights = (_weight_bytes(QKV_A, HIDDEN, proj) + _weight_bytes(HEADS * QK, Q_LORA, proj)
               + _weight_bytes(HEADS * (NOPE + V_DIM), KV_LORA, proj) + _weight_bytes(HIDDEN, HEADS * V_DIM, proj))
    flops = 2.0 * t * n_proj + 2.0 * HEADS * (t * (t + 1) // 2) * (QK + V_DIM)
    if case["ffn"] == "dense":
        weights += _weight_bytes(2 * DENSE_INTER, HIDDEN, proj) + _weight_bytes(HIDDEN, DENSE_INTER, proj)
        flops += 2.0 * t * 3 * DENSE_INTER * HIDDEN
    else:
        eb, ef = _experts(t)
        weights += eb + EXPERTS * HIDDEN * 2
        flops += ef + 2.0 * t * EXPERTS * HIDDEN
    return {"bytes": weights + 10 * t * HIDDEN * 2, "flops": flops}


def tolerance(case: dict):
    """About four times what was measured between two evaluations of a case on one B200: its sums in
    64 bits (prologue, the expert products), its reductions cut differently (the K range of the
    few-row projections, the attention schedules)."""
    kind = case["kind"]
    if kind == "swiglu_quant":
        return "exact"                                   # codes and scales are defined bit for bit
    if kind == "prologue":
        # 1e-5 over thousands of rows, but one last bit among the 64 values of a single k_pe row is 1e-3
        return {"rel": 1.0e-3, "max": 0.032}
    if kind == "indexer":
        # a last bit of the projected key flips 2e-3 of its e4m3 codes, near-ties 1e-4 of the mask
        return {"rel": 1.3e-3, "max": 0.025, "differ": 9.0e-3}
    if kind == "moe":
        return {"rel": 4.0e-3, "max": 0.08}              # 9.5e-4: NVFP4 codes flipped by a last bit of h
    if kind == "decode":
        # 3.8e-3: the picked positions that near-ties decide, else the order of the projections' sums
        return {"rel": 1.5e-2, "max": 0.08, "differ": 1.0e-3}
    return {"rel": 1.2e-2, "max": 0.16}                  # 3.1e-3, FP8 and NVFP4 codes flipped by a last bit
