"""Performance cases of the framework: the calls that a serving engine and a user of the quantizer make.

Each case is one layer's call(s) through the public Python entry points: ``TurboQuantPagedAttention`` (cache write,
decode, shared and causal queries, bulk dequantization) and ``TurboQuantMSE``.  ``listed`` holds the fixed cases,
``draw`` gives more of the same ranges.  Caches are filled by the cache write itself from N(0, 1) keys and values, pages
are a random permutation, and sequence lengths are log-uniform between two bounds (the benchmark's mixed batch), so
that a batch is ragged unless both bounds are equal.
"""
from __future__ import annotations

import math
import random

import torch

from turboquant_b200 import TurboQuantMSE, TurboQuantPagedAttention
from turboquant_b200.paged_attention import kv_cache_shape

PAGE = 16
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
# (query heads, KV heads) by head size, from the package's model presets
HEADS = {128: ((32, 8), (16, 8), (40, 8), (64, 8), (32, 4), (56, 8), (32, 32), (40, 40)),
         96: ((32, 8), (32, 32)), 64: ((16, 8),), 256: ((16, 8), (8, 4))}
MOST_TOKEN_HEADS = 8 << 20      # cached tokens x KV heads of the largest listed case


def _step(name, batch, lo, hi, heads=(32, 8), head_size=128, dtype="bf16", lens_seed=3):
    return {"name": name, "kind": "step", "batch": batch, "len_lo": lo, "len_hi": hi, "lens_seed": lens_seed,
            "q_heads": heads[0], "kv_heads": heads[1], "head_size": head_size, "dtype": dtype}


def listed():
    return [
        # One decode step of one layer: the new tokens of all sequences are quantized into the cache, then attended.
        # A single user's chat with a short context: latency of the calls is everything.
        _step("step_b1_ctx1024", 1, 1024, 1024, dtype="fp16"),
        # An ordinary serving batch, ragged short to medium contexts, five query heads per KV head.
        _step("step_b32_ragged", 32, 128, 4096, heads=(40, 8)),
        # The long-context batch of the benchmark's headline.
        _step("step_b8_ctx32768", 8, 32768, 32768),
        # The benchmark's mixed batch: lengths over a factor of 256 in one call.
        _step("step_b64_mixed", 64, 512, 131072),
        # The small and the large head size of the presets, ragged batches.
        _step("step_b16_head64", 16, 1000, 16000, heads=(16, 8), head_size=64),
        _step("step_b8_head256", 8, 1000, 16000, heads=(16, 8), head_size=256),
        # Cache write of a long prompt: K has 1 % of its channels as outliers.
        {"name": "write_prompt_32768", "kind": "write", "tokens": 32768, "skipped": 0, "kv_heads": 8, "head_size": 128, "dtype": "bf16"},
        # Cache write of one chunk of a chunked prefill, padded to the engine's bucket (slots of -1 are skipped).
        {"name": "write_chunk_2000", "kind": "write", "tokens": 2048, "skipped": 48, "kv_heads": 32, "head_size": 96, "dtype": "fp16"},
        # Verification step of speculative decoding / a short continuing chunk: causal queries over the cache.
        {"name": "causal_b8_q8_ctx32768", "kind": "causal", "batch": 8, "queries": 8, "len_lo": 32768, "len_hi": 32768, "lens_seed": 3,
         "q_heads": 32, "kv_heads": 8, "head_size": 128, "dtype": "bf16"},
        # Eight queries that share one sequence of a million tokens.
        {"name": "shared_b1_q8_ctx1m", "kind": "shared", "batch": 1, "queries": 8, "len_lo": 1 << 20, "len_hi": 1 << 20, "lens_seed": 3,
         "q_heads": 32, "kv_heads": 8, "head_size": 128, "dtype": "bf16"},
        # Cached context of a continuing prefill back to dense K / V for a varlen attention kernel.
        {"name": "dequant_b8_ctx8192", "kind": "dequant", "batch": 8, "len_lo": 5000, "len_hi": 13000, "lens_seed": 3,
         "kv_heads": 8, "head_size": 128, "dtype": "bf16"},
        # The quantizer on its own: vectors to codes and norms and back (accuracy studies, weights of other tools).
        {"name": "quantizer_65536x128", "kind": "quantizer", "rows": 65536, "head_size": 128, "bits": 4, "dtype": "fp16"},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def _draw_lengths(rng, longest, batch, kv_heads):
    """Bounds of a ragged batch whose cached tokens x KV heads stay within the largest listed case."""
    hi = _log_int(rng, PAGE, max(PAGE, min(longest, MOST_TOKEN_HEADS // (batch * kv_heads))))
    return {"len_lo": max(1, hi // rng.choice((1, 1, 4, 32, 256))), "len_hi": hi, "lens_seed": rng.randrange(1 << 20)}


def draw(rng):
    kind = rng.choices(("step", "write", "causal", "shared", "dequant", "quantizer"), (50, 15, 10, 5, 10, 10))[0]
    dtype = rng.choice(("bf16", "bf16", "fp16"))
    if kind == "quantizer":
        return {"kind": kind, "rows": _log_int(rng, 1, 131072), "head_size": rng.choice((64, 96, 128, 128, 256)),
                "bits": rng.choice((2, 3, 4, 4)), "dtype": rng.choice(("bf16", "fp16", "fp32"))}
    if kind in ("causal", "shared"):      # the geometries whose queries go through one pass over the KV
        head_size = rng.choice((128, 128, 128, 96))
        q_heads, kv_heads = rng.choice([h for h in HEADS[head_size] if h[1] in (2, 4, 8, 16)])
        queries = rng.randint(2, min(8, 32 // (q_heads // kv_heads)))
        batch = _log_int(rng, 1, 32) if kind == "causal" else _log_int(rng, 1, 4)
        case = {"kind": kind, "batch": batch, "queries": queries, **_draw_lengths(rng, 1 << 20, batch, kv_heads)}
        case["len_lo"] = max(case["len_lo"], queries)
        return {**case, "q_heads": q_heads, "kv_heads": kv_heads, "head_size": head_size, "dtype": dtype}
    head_size = rng.choice((128, 128, 128, 128, 96, 64, 256))
    q_heads, kv_heads = rng.choice(HEADS[head_size])
    if kind == "write":
        tokens = _log_int(rng, 1, 32768 * 8 // max(8, kv_heads) * 128 // max(128, head_size))
        return {"kind": kind, "tokens": tokens, "skipped": tokens // 40 if rng.random() < 0.3 else 0, "kv_heads": kv_heads,
                "head_size": head_size, "dtype": dtype}
    if kind == "dequant":
        batch = _log_int(rng, 1, 16)
        longest = 65536 * 8 // kv_heads * 128 // max(128, head_size) // batch
        return {"kind": kind, "batch": batch, **_draw_lengths(rng, longest, batch, kv_heads), "kv_heads": kv_heads,
                "head_size": head_size, "dtype": dtype}
    batch = _log_int(rng, 1, 64)
    return {"kind": kind, "batch": batch, **_draw_lengths(rng, 131072, batch, kv_heads), "q_heads": q_heads, "kv_heads": kv_heads,
            "head_size": head_size, "dtype": dtype}


def _lengths(case):
    """Sequence lengths of the batch, log-uniform in [len_lo, len_hi]; the longest is len_hi."""
    rng = random.Random(case["lens_seed"])
    lens = [_log_int(rng, case["len_lo"], case["len_hi"]) for _ in range(case["batch"])]
    lens[rng.randrange(len(lens))] = case["len_hi"]
    return lens


def _filled_cache(attn, pages, dtype, gen):
    """A cache of ``pages`` pages whose every slot holds a quantized N(0, 1) key and value."""
    H, D = attn.num_kv_heads, attn.head_size
    cache = torch.zeros(kv_cache_shape(pages, PAGE, H, D), dtype=torch.uint8, device="cuda")
    chunk = max(PAGE, (1 << 26) // (H * D))
    for at in range(0, pages * PAGE, chunk):
        n = min(chunk, pages * PAGE - at)
        k = torch.randn(n, H, D, generator=gen, dtype=dtype, device="cuda")
        v = torch.randn(n, H, D, generator=gen, dtype=dtype, device="cuda")
        attn.write(k, v, cache, torch.arange(at, at + n, device="cuda"))
    return cache


def _paged_batch(case, attn, gen):
    """Filled cache, block table (pages in a random permutation), lengths and the slot of every sequence's last token."""
    lens = torch.tensor(_lengths(case), dtype=torch.int64, device="cuda")
    pages = (lens + PAGE - 1) // PAGE
    total, longest = int(pages.sum()), int(pages.max())
    table = torch.zeros(case["batch"], longest, dtype=torch.int32, device="cuda")
    table[torch.arange(longest, device="cuda")[None, :] < pages[:, None]] = \
        torch.randperm(total, generator=gen, device="cuda").to(torch.int32)
    last = lens - 1
    slots = table.gather(1, (last // PAGE)[:, None])[:, 0].long() * PAGE + last % PAGE
    cache = _filled_cache(attn, total, DTYPES[case["dtype"]], gen)
    return {"cache": cache, "block_table": table, "seq_lens": lens.to(torch.int32), "slots": slots}


def prepare(case, seed):
    gen = torch.Generator("cuda")
    gen.manual_seed(seed)
    kind, D, dtype = case["kind"], case["head_size"], DTYPES[case["dtype"]]

    def normal(*shape):
        return torch.randn(*shape, generator=gen, dtype=dtype, device="cuda")

    if kind == "quantizer":
        return {"kind": kind, "quantizer": TurboQuantMSE(D, case["bits"], device="cuda"), "x": normal(case["rows"], D)}
    H, Hq = case["kv_heads"], case.get("q_heads", case["kv_heads"])
    attn = TurboQuantPagedAttention(Hq, D, 1.0 / math.sqrt(D), H)
    state = {"kind": kind, "attn": attn, "dtype": dtype}
    if kind == "write":
        T = case["tokens"]
        pages = (T + PAGE - 1) // PAGE
        k, v = normal(T, H, D), normal(T, H, D)
        k[..., torch.randperm(D, generator=gen, device="cuda")[: max(1, round(0.01 * D))]] *= 20.0
        order = torch.randperm(pages, generator=gen, device="cuda")
        t = torch.arange(T, device="cuda")
        slots = order[t // PAGE] * PAGE + t % PAGE
        if case["skipped"]:
            slots[T - case["skipped"]:] = -1
        cache = torch.zeros(kv_cache_shape(pages, PAGE, H, D), dtype=torch.uint8, device="cuda")
        return {**state, "cache": cache, "k": k, "v": v, "slots": slots}
    state.update(_paged_batch(case, attn, gen))
    B = case["batch"]
    if kind == "dequant":
        lens = state["seq_lens"]
        cu = torch.zeros(B + 1, dtype=torch.int32, device="cuda")
        cu[1:] = torch.cumsum(lens, 0)
        return {**state, "cu_seqlens": cu, "total": int(cu[-1])}
    shape = (B, Hq, D) if kind == "step" else (B, case["queries"], Hq, D)
    state.update(q=normal(*shape), out=torch.empty(*shape, dtype=dtype, device="cuda"))
    if kind == "step":
        state.update(k=normal(B, H, D), v=normal(B, H, D))
    return state


def run(s):
    kind = s["kind"]
    if kind == "step":
        s["attn"].write(s["k"], s["v"], s["cache"], s["slots"])
        return s["attn"].decode(s["q"], s["cache"], s["block_table"], s["seq_lens"], s["out"]), s["cache"]
    if kind == "write":
        s["attn"].write(s["k"], s["v"], s["cache"], s["slots"])
        return s["cache"]
    if kind == "causal":
        return s["attn"].decode_causal(s["q"], s["cache"], s["block_table"], s["seq_lens"], s["out"])
    if kind == "shared":
        return s["attn"].decode_shared(s["q"], s["cache"], s["block_table"], s["seq_lens"], s["out"])
    if kind == "dequant":
        return s["attn"].dequant_cached(s["cache"], s["block_table"], s["seq_lens"], s["cu_seqlens"], s["total"], s["dtype"])
    packed, norms = s["quantizer"].quantize(s["x"])
    return packed, norms, s["quantizer"].dequantize(packed, norms)


def work(case):
    kind, D = case["kind"], case["head_size"]
    padded = 1 << (D - 1).bit_length()
    size = 4 if case["dtype"] == "fp32" else 2
    butterflies = padded * int(math.log2(padded))      # additions of one rotation
    if kind == "quantizer":
        n, codes = case["rows"], padded * case["bits"] / 8
        # x in, codes and fp32 norms out; codes and norms in, fp32 vectors out
        return {"bytes": n * (D * size + 2 * (codes + 4) + 4 * D), "flops": n * (2 * butterflies + 6 * padded)}
    H = case["kv_heads"]
    row = padded // 2 + 2                               # codes and one fp16 norm
    if kind == "write":
        n = 2 * H * (case["tokens"] - case["skipped"])
        return {"bytes": n * (D * size + row) + 8 * case["tokens"], "flops": n * (butterflies + 3 * padded)}
    tokens = sum(_lengths(case))
    cached = 2 * H * row * tokens
    if kind == "dequant":
        return {"bytes": cached + 2 * H * tokens * D * size, "flops": 2 * H * tokens * (butterflies + 2 * padded)}
    queries = case["batch"] * case.get("queries", 1)
    bytes_ = cached + 2 * queries * case["q_heads"] * D * size
    if kind == "step":
        bytes_ += 2 * case["batch"] * H * (D * size + row)
    return {"bytes": bytes_, "flops": 4 * case["q_heads"] * padded * tokens * case.get("queries", 1)}


def tolerance(case):
    """Codes, norms and cache bytes are whole values and equal.  Attention outputs: probabilities and dequantized values
    are 16-bit operands with fp32 sums, and the result is rounded to its type.  Dequantized rows: 32-bit sums, rounded."""
    kind = case["kind"]
    if kind == "write":
        return "exact"
    if kind == "quantizer":
        return {"rel": 1e-5}
    if kind == "dequant":
        return {"rel": 4e-3 if case["dtype"] == "bf16" else 5e-4}
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 4e-3}
