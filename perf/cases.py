"""The work that users of turboquant_b200 have it do, one layer at a time, as timed cases.

A case is one pass of one attention layer through the package's public entry points:

* "prefill":  rotary embedding (`rope`, where the model has one), `compress_kv`, `fused_attention` -- what an adapter
  of a patched model does with the projections of a prompt;
* "generate": `CompressedKVCache.append` of the new tokens, then `attend` of their queries over everything cached -- one
  token per sequence (a generation step) or a chunk of a prompt or of a next turn;
* "inspect":  `compress` of both sides, `asymmetric_attention_scores` of the last query of every head and `decompress`
  -- what the quality harness and users who look at the estimator do.

Shapes are those of the repository's configurations: LLaMA-3-8B (32 query heads, 8 KV heads, head_dim 128), Qwen2.5-3B
(16 / 2 / 128), DeepSeek-7B (32 / 32 / 128) and GPT-2-small (12 / 12 / 64).  Inputs are standard normal with four outlier
channels per key head (x 8), the distribution of the benchmark, in the layouts that the projections leave behind.
"""

from __future__ import annotations

import math
import os
import random
import sys

import torch

_PACKAGES = os.path.join(os.getcwd(), "transformers-turboquant_b200")
if _PACKAGES not in sys.path:
    sys.path.insert(0, _PACKAGES)

import turboquant_b200 as tq  # noqa: E402

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
_SHAPES = {"llama8b": (32, 8, 128), "qwen3b": (16, 2, 128), "deepseek7b": (32, 32, 128), "gpt2": (12, 12, 64)}
_ROPE_BASE = {"llama8b": 500000.0, "qwen3b": 1000000.0, "deepseek7b": 10000.0}


def listed():
    return [
        # a generation step of one chat: latency and launches count, there are few bytes to read
        _case("step_1x2000", "generate", "llama8b", batch=1, cached=2000, tokens=1),
        # a generation step of a small batch over long contexts (the decode benchmark's shape)
        _case("step_8x32767", "generate", "llama8b", batch=8, cached=32767, tokens=1),
        # a serving batch of a multi-head model, prompts of several lengths padded on the left
        _case("step_padded_mha_16x4000", "generate", "deepseek7b", batch=16, cached=4000, tokens=1, bits=2, padded=True),
        # text generation with GPT-2, the one family of head_dim 64
        _case("step_gpt2_4x700", "generate", "gpt2", batch=4, cached=700, tokens=1),
        # the next turn of a chat, or a chunk of a long prompt: a few hundred new tokens behind a long prefix
        _case("chunk_1x8000+300", "generate", "llama8b", batch=1, cached=8000, tokens=300),
        # one medium prompt through the smallest GQA model, at 4 bits
        _case("prefill_qwen_1x2048", "prefill", "qwen3b", batch=1, tokens=2048, bits=4),
        # a layer of the LLaMA-8B prefill configuration (batch 8, 4096 tokens)
        _case("prefill_llama_8x4096", "prefill", "llama8b", batch=8, tokens=4096),
        # the operator benchmark's shape: the longest prompts of the configurations, batched
        _case("prefill_llama_4x8192", "prefill", "llama8b", batch=4, tokens=8192),
        # a padded batch of ragged prompts in fp16, with the boolean mask that the sdpa path of HF hands over
        _case("prefill_padded_fp16_6x777", "prefill", "llama8b", batch=6, tokens=777, dtype="fp16", padded=True),
        # GPT-2-small in full precision, the configuration of the reference's own end-to-end check
        _case("prefill_gpt2_fp32_1x1024", "prefill", "gpt2", batch=1, tokens=1024, dtype="fp32"),
        # GPT-2-small, a batch of full contexts in bf16
        _case("prefill_gpt2_8x1024", "prefill", "gpt2", batch=8, tokens=1024),
        # the quality harness on one layer: encode both sides, score the last query, decode the values
        _case("inspect_qwen_1x8192", "inspect", "qwen3b", batch=1, tokens=8192),
    ]


def _case(name, kind, shape, batch, tokens, cached=0, bits=3, dtype="bf16", padded=False):
    case = {"name": name} if name else {}
    return {**case, "kind": kind, "shape": shape, "batch": batch, "cached": cached, "tokens": tokens, "bits": bits,
            "dtype": dtype, "padded": padded}


def _between(rng, low, high):
    """A whole number between low and high, spread evenly over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng: random.Random):
    kind = rng.choice(["generate", "generate", "generate", "prefill", "prefill", "prefill", "inspect"])
    shape = rng.choice(["llama8b", "llama8b", "qwen3b", "deepseek7b", "gpt2"])
    bits = rng.choice([2, 3, 3, 4])
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16", "fp32"]) if kind != "inspect" else rng.choice(["bf16", "fp32"])
    padded = kind != "inspect" and rng.random() < 0.2
    longest = 1024 if shape == "gpt2" else 32768
    # score elements of one pass: the largest listed case has 4.3e9; fp32 costs over ten times as much, and tiles of
    # 64 query rows
    limit, tile = {"bf16": (4e9, 1), "fp16": (4e9, 1), "fp32": (1e8, 64)}[dtype]
    heads, kv_heads, _ = _SHAPES[shape]
    while True:
        batch = _between(rng, 1, 32)
        if kind == "generate":
            cached = _between(rng, 16, longest)
            tokens = 1 if rng.random() < 0.6 else _between(rng, 2, 1024)
        else:
            cached, tokens = 0, _between(rng, 16, longest)
        total = cached + tokens
        if total > longest or batch * total > 8 * 32768:
            continue
        if kind == "inspect" and batch * kv_heads * total > 1e6:
            continue
        if kind != "inspect" and batch * heads * max(tokens, tile) * (cached + tokens / 2) > limit:
            continue
        if padded and batch * tokens * total > 1.5e8:  # the mask is a matrix
            continue
        return _case("", kind, shape, batch, tokens, cached, bits, dtype, padded)


def _normal(gen, *shape):
    return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float32)


def _outliers(gen, case):
    """Factors of the key channels of every head: four of them 8, the others 1."""
    _, Hkv, D = _SHAPES[case["shape"]]
    channels = torch.rand(Hkv, D, generator=gen, device="cuda").topk(4, dim=-1).indices
    return torch.ones(Hkv, D, device="cuda").scatter_(1, channels, 8.0)


def _projections(gen, case, gain):
    """Queries, keys and values [B, H, S, D] as a layer's projections leave them: views of [B, S, H, D] for the
    models with separate projections, slices of one fused projection for GPT-2."""
    Hq, Hkv, D = _SHAPES[case["shape"]]
    B, tokens, dtype = case["batch"], case["tokens"], _DTYPES[case["dtype"]]
    if case["shape"] == "gpt2":
        fused = _normal(gen, B, tokens, 3, Hq, D)
        fused[:, :, 1] *= gain
        parts = fused.to(dtype).unbind(2)
    else:
        parts = [_normal(gen, B, tokens, Hq, D).to(dtype), (_normal(gen, B, tokens, Hkv, D) * gain).to(dtype),
                 _normal(gen, B, tokens, Hkv, D).to(dtype)]
    return [t.transpose(1, 2) for t in parts]


def _rotary_tables(case, tokens):
    D = _SHAPES[case["shape"]][2]
    inv = _ROPE_BASE[case["shape"]] ** (-torch.arange(0, D, 2, device="cuda", dtype=torch.float32) / D)
    angle = torch.arange(tokens, device="cuda", dtype=torch.float32)[:, None] * inv
    angle = torch.cat([angle, angle], dim=-1)[None]
    return angle.cos().to(_DTYPES[case["dtype"]]), angle.sin().to(_DTYPES[case["dtype"]])


def _padding_mask(gen, case):
    """[B, 1, S_new, S_all], True = visible: causal, and only real tokens.  Prompts are padded on the right, a cache
    that generates is padded on the left."""
    B, new, total = case["batch"], case["tokens"], case["cached"] + case["tokens"]
    lengths = (total * (0.5 + 0.5 * torch.rand(B, generator=gen, device="cuda"))).long().clamp(min=1)
    if case["cached"]:
        lengths = lengths.clamp(min=min(new + 1, total))
    position = torch.arange(total, device="cuda")
    real = position >= (total - lengths)[:, None] if case["cached"] else position < lengths[:, None]
    causal = position <= torch.arange(case["cached"], total, device="cuda")[:, None]
    return (causal & real[:, None, :])[:, None]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    Hq, Hkv, D = _SHAPES[case["shape"]]
    layer_seed = 42 + int(seed) % 32
    state = {"case": case, "kc": tq.TurboQuantCompressorV2(D, case["bits"], seed=layer_seed, device="cuda"),
             "vc": tq.TurboQuantCompressorMSE(D, case["bits"], seed=layer_seed + 10000, device="cuda"), "mask": None}
    gain = _outliers(gen, case)
    state["q"], state["k"], state["v"] = _projections(gen, case, gain)
    if case["padded"]:
        state["mask"] = _padding_mask(gen, case)
    if case["kind"] == "inspect":
        # the harness takes the last key of every KV head for a query
        state["q"] = state["k"][:, :, -1:, :]
    if case["kind"] == "prefill" and case["shape"] in _ROPE_BASE:
        state["rotary"] = _rotary_tables(case, case["tokens"])
    if case["kind"] == "generate":
        total = case["cached"] + case["tokens"]
        cache = tq.CompressedKVCache(state["kc"], state["vc"], case["batch"], Hkv, total + total // 8 + 16)
        dtype = _DTYPES[case["dtype"]]
        for at in range(0, case["cached"], 8192):
            chunk = (case["batch"], Hkv, min(8192, case["cached"] - at), D)
            cache.append((_normal(gen, *chunk) * gain[:, None]).to(dtype), _normal(gen, *chunk).to(dtype))
        state["cache"] = cache
    return state


def run(state):
    case, q, k, v, kc, vc = (state[n] for n in ("case", "q", "k", "v", "kc", "vc"))
    if case["kind"] == "prefill":
        if "rotary" in state:
            q, k = tq.rope(q, k, *state["rotary"])
        ck, cv = tq.compress_kv(k, v, kc, vc)
        out = tq.fused_attention(q, ck, cv, kc, vc, causal=True, attention_mask=state["mask"])
        return {"out": out, "keys": _arrays(ck), "values": _arrays(cv)}
    if case["kind"] == "generate":
        cache = state["cache"]
        cache.length = case["cached"]  # drops what the pass before appended
        cache.append(k, v)
        out = cache.attend(q, causal=True, attention_mask=state["mask"])
        return {"out": out, "cache": [cache.key_indices, cache.key_signs, cache.key_norms, cache.key_residual_norms,
                                      cache.value_indices, cache.value_norms]}
    ck, cv = kc.compress(k), vc.compress(v)
    scores = kc.asymmetric_attention_scores(q, ck)
    return {"scores": scores, "decoded": vc.decompress(cv), "keys": _arrays(ck), "values": _arrays(cv)}


def _arrays(compressed):
    return {name: t for name, t in compressed.items() if isinstance(t, torch.Tensor)}


def work(case):
    Hq, Hkv, D = _SHAPES[case["shape"]]
    B, new, old, size = case["batch"], case["tokens"], case["cached"], _DTYPES[case["dtype"]].itemsize
    # key indices, signs and two norms, value indices and a norm
    packed = D * (case["bits"] - 1) // 8 + D // 8 + 4 + D * case["bits"] // 8 + 2
    vectors = B * Hkv * new
    flops = vectors * 6 * D * D  # rotation and sketch of a key, rotation of a value
    bytes_ = vectors * (2 * D * size + packed)  # new keys and values in, packed bytes out
    if case["kind"] == "inspect":
        bytes_ += vectors * (4 * D + 4)  # decoded values and scores out
        return {"bytes": bytes_, "flops": flops + vectors * (2 * D * D + 4 * D)}
    bytes_ += 2 * B * Hq * new * D * size + B * Hkv * old * packed  # queries in, output out, the cache in
    if case["padded"]:
        bytes_ += B * new * (old + new)
    if case["kind"] == "prefill" and case["shape"] in _ROPE_BASE:
        bytes_ += 2 * new * D * size
    pairs = B * Hq * (new * old + new * (new + 1) // 2)
    # rotated and sketched query against a key, probability times value; the rotations of a query and of an output row
    return {"bytes": bytes_, "flops": flops + pairs * 6 * D + B * Hq * new * 6 * D * D}


def tolerance(case):
    """About four times what correct evaluations of the same path were seen to differ by.  An index or a sign whose
    coordinate lies within rounding of its boundary falls either way; one of them in the first keys of a causal head
    moves that head's first outputs by a large part of their value, hence the wide `max` beside a narrow `rel`.
      * attention of 16-bit inputs against the same bytes attended in fp32: rel 5e-3 (the repository's bound is 1e-2);
      * fp32 against an evaluation of everything in fp64: rel 2e-3, all of it from a flipped sign or value index;
      * encode and decode of bf16 inputs against the fp32 kernels: rel 1e-3.
    Bytes: bf16 inputs are rotated on the tensor cores (3e-4 of the sign bytes, 2e-5 of the index bytes differ from
    the fp32 kernels'), fp16 and fp32 inputs in fp32 (1e-5 of the sign bytes differ from fp64)."""
    if case["kind"] == "inspect":
        rel = 4e-3
    else:
        rel = 6e-3 if case["dtype"] == "fp32" else 1e-2
    return {"rel": rel, "max": 0.99, "differ": 1.2e-3 if case["dtype"] == "bf16" else 5e-5}
