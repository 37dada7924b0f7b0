"""The work this package is measured on: cases over the range of shapes its users run.

``listed()`` are the fixed cases, ``draw(rng)`` makes further ones of the same ranges.  A case is a
dict of plain values; ``prepare`` builds its inputs on the GPU, ``run`` makes one pass through the
public entry points, ``work`` counts what a pass cannot do without and ``tolerance`` says how far
another correct implementation of the same precision may be from the result.
"""
import math

import torch

from flash_colreduce_b200 import flash_colreduce, topk_columns, valid_scores

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}

# No drawn case does more multiply-adds than the largest listed one (8 heads of 131072^2, causal,
# d = 128) or reads more than the largest listed decode batch (16 x 32 heads of 16384 keys, d = 128).
_MAX_SCORES_D = 8 * 131072 * 131073 // 2 * 128
_MAX_BYTES = 16 * 32 * (16384 + 64) * 128 * 2


def _case(name, b, h, m, n, d, causal, reduction, dtype="fp16", layout="bhmd", values="normal", scale=0.0):
    """One ``flash_colreduce`` call.  ``layout``: "bhmd" contiguous, "bmhd" as the transposed view of a
    projection's (B, M, H, D) output.  ``values``: "normal" i.i.d. N(0, 1), "sinks" with four
    attention-sink keys and a block of visual tokens.  ``scale`` 0: the default 1 / sqrt(d)."""
    return {"name": name, "op": "colreduce", "b": b, "h": h, "m": m, "n": n, "d": d, "causal": causal,
            "reduction": reduction, "dtype": dtype, "layout": layout, "values": values, "scale": scale}


def _topk(name, rows, n, k, dtype="fp16"):
    return {"name": name, "op": "topk", "rows": rows, "n": n, "k": k, "dtype": dtype}


def listed():
    return [
        # One short text sequence through a small encoder: nothing but latency.
        _case("square_256_d64", 2, 4, 256, 256, 64, False, "sum"),
        # A batch of short sequences, one head per SM: small work items, set-up counts.
        _case("batch_512_d64_mean", 8, 16, 512, 512, 64, False, "mean"),
        # A block of draft or suffix tokens scored against a 4096-key context in one layer.
        _case("block_128x4096_max", 1, 32, 128, 4096, 128, True, "max"),
        # KV-cache eviction in a serving batch: the last 64 queries score 16384 cached keys.
        _case("window_64x16384_batch16", 16, 32, 64, 16384, 128, True, "sum"),
        # The same at every decode step: one query per sequence, ragged context, K read once.
        _case("token_1x8191_batch32_bf16", 32, 32, 1, 8191, 128, True, "sum", dtype="bf16"),
        # A 512-token chunk of a long prompt against the 32768 keys so far.
        _case("chunk_512x32768_bf16_mean", 1, 32, 512, 32768, 128, True, "mean", dtype="bf16"),
        # A batch of image-encoder sequences without a mask.
        _case("batch16_1024", 16, 32, 1024, 1024, 128, False, "sum"),
        # A prompt of odd length, head dimension 80, q and k as a projection leaves them (B, M, H, D).
        _case("ragged_3001_d80_bmhd", 2, 20, 3001, 3001, 80, True, "mean", dtype="bf16", layout="bmhd"),
        # fp32 inputs, multiplied as TF32.
        _case("fp32_2048_d64", 4, 16, 2048, 2048, 64, True, "sum", dtype="fp32"),
        # Visual-token pruning over a long multi-modal prompt: sinks and a flat block of visual keys.
        _case("vlm_8192_mean", 4, 32, 8192, 8192, 128, True, "mean", values="sinks"),
        # The consumer's selection step on such scores: a quarter of 8192 keys of every head.
        _topk("topk_128x8192_k2048", 128, 8192, 2048),
        # One GPU's eight heads of the long-context problem.
        _case("long_131072_8heads", 1, 8, 131072, 131072, 128, True, "sum"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["small", "block", "token", "chunk", "square", "square", "long", "topk"])
    if family == "topk":
        n = _log_uniform(rng, 500, 131072)
        rows = min(_log_uniform(rng, 16, 4096), (1 << 28) // n)
        k = max(1, min(n, int(n * rng.uniform(0.05, 0.6))))
        case = _topk("", rows, n, k, rng.choice(["fp16", "bf16", "fp32"]))
        del case["name"]
        return case
    b, h = _log_uniform(rng, 1, 16), rng.choice([4, 8, 12, 16, 20, 32])
    d = rng.choice([64, 64, 80, 96, 128, 128, 128, 256])
    dtype = rng.choice(["fp16", "fp16", "bf16", "bf16", "fp32"])
    causal = rng.random() < 0.6
    if family == "small":
        m = _log_uniform(rng, 64, 768)
        n = m if rng.random() < 0.6 else _log_uniform(rng, 64, 768)
    elif family == "token":
        m, n, causal = rng.choice([1, 1, 2, 4]), _log_uniform(rng, 1024, 32768), True
        b *= 2
    elif family == "block":
        m, n, causal = _log_uniform(rng, 5, 128), _log_uniform(rng, 1024, 65536), True
    elif family == "chunk":
        m, n, causal = _log_uniform(rng, 129, 1024), _log_uniform(rng, 4096, 131072), True
    elif family == "square":
        m = n = _log_uniform(rng, 768, 16384)
    else:
        m = n = _log_uniform(rng, 16384, 131072)
        b, h, causal = 1, rng.choice([1, 2, 4, 8]), True
    if rng.random() < 0.5 and m > 64:  # whole multiples of 64 and odd lengths in equal parts
        m, n = m // 64 * 64, max(64, n // 64 * 64)
    if dtype == "fp32":
        d = min(d, 128)
    size = 4 if dtype == "fp32" else 2
    while b * h > 1 and (valid_scores(b, h, m, n, causal) * d > _MAX_SCORES_D // 2
                         or b * h * (m + n) * d * size > _MAX_BYTES // 2):
        b, h = (b // 2, h) if b > 1 else (1, h // 2)
    case = _case("", b, h, m, n, d, causal, rng.choice(["sum", "mean", "max"]), dtype=dtype,
                 layout=rng.choice(["bhmd", "bhmd", "bmhd"]), values="sinks" if n >= 4096 and rng.random() < 0.3 else "normal",
                 scale=0.0 if rng.random() < 0.8 else round(rng.uniform(0.5, 1.5) / math.sqrt(d), 4))
    del case["name"]
    return case


def _operand(case, rows, gen):
    b, h, d = case["b"], case["h"], case["d"]
    shape = (b, h, rows, d) if case["layout"] == "bhmd" else (b, rows, h, d)
    x = torch.randn(shape, generator=gen, dtype=_DTYPES[case["dtype"]], device="cuda")
    return x if case["layout"] == "bhmd" else x.transpose(1, 2)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["op"] == "topk":
        # Column scores of an attention head: heavy-tailed, a few sinks far above the rest, rounded to
        # the score's type (so that ties occur).
        x = torch.randn((case["rows"], case["n"]), generator=gen, dtype=torch.float32, device="cuda").exp_().div_(case["n"])
        x[:, :4] *= 1000.0
        return {"case": case, "scores": x.to(_DTYPES[case["dtype"]])}
    q = _operand(case, case["m"], gen)
    k = _operand(case, case["n"], gen)
    if case["values"] == "sinks":
        # the first four keys are attention sinks, three quarters of the keys a flat visual block
        n = case["n"]
        k[:, :, :4] *= 8.0
        k[:, :, n // 16 : n // 16 + 3 * n // 4] *= 0.5
    return {"case": case, "q": q, "k": k}


def run(state):
    case = state["case"]
    if case["op"] == "topk":
        return topk_columns(state["scores"], case["k"])
    return flash_colreduce(state["q"], state["k"], case["reduction"], is_causal=case["causal"],
                           scale=case["scale"] or None)


def work(case):
    size = 4 if case["dtype"] == "fp32" else 2
    if case["op"] == "topk":
        # every score once, an int64 position and a score for each selected key
        return {"bytes": case["rows"] * (case["n"] * size + case["k"] * (8 + size)), "flops": 0}
    b, h, m, n, d = (case[x] for x in ("b", "h", "m", "n", "d"))
    # A column's sum needs every row's normaliser first, which needs every score of the row: the scores
    # are computed twice (2*d flops each time) because the matrix of them is never stored.
    return {"bytes": b * h * ((m + n) * d + n) * size, "flops": 4 * d * valid_scores(b, h, m, n, case["causal"])}


def tolerance(case):
    if case["op"] == "topk":
        return "exact"
    # Measured against the definition in 64 bits over these ranges: fp16 results lie 1.9e-4 to 3.5e-4 away
    # and bf16 results 0.8e-3 to 1.9e-3, all of it the one rounding to the result's type.  Two correct
    # results round apart only where their fp32 sums straddle a rounding boundary (up to 2.5e-5 seen).
    if case["dtype"] == "fp16":
        return {"rel": 4e-4}
    if case["dtype"] == "bf16":
        return {"rel": 2.5e-3}
    # fp32 inputs: the operands are TF32 (10 mantissa bits), 1.4e-4 for sums and more for single maxima
    return {"rel": 1e-3}
