"""The work that a serving or training program has this package do, as cases that can be timed.

Each case is a dict of plain values; `prepare` makes what the program has in hand before the call, `run` is one pass
through the public entry points, `work` what that pass cannot do without.  The kinds of work:

  attend   top-k sparse MLA forward on a bf16 latent cache (`sparse_mla_fwd`): decode of a few tokens over a long
           context, or prefill of a chunk of tokens that see a causal prefix.
  step     one decode step on the paged FP8 latent cache: append the new rows (`kv_cache_write_fp8`), choose the
           positions (`topk_indices`), attend to them (`sparse_mla_fwd_paged`).
  fill     the cache write of a prefill (`kv_cache_write_fp8`).
  select   index lists of a prefill from its score matrix (`topk_indices`).
  merge    results of the ranks that each hold a slice of the context (`sparse_mla_merge`).
  matmul   bf16 projection (`matmul`).
  matmul8  block-scaled FP8 projection (`matmul_fp8_blockscaled`).
"""
import math

import torch

import flagtree_b200 as ft

DEV = "cuda:0"
D_QK, D_V, PAGE = 576, 512, 64
SM_SCALE = 192 ** -0.5


def listed():
    return [
        # one sequence, one new token: the latency of a single decode call
        {"name": "attend_1_token", "kind": "attend", "tokens": 1, "heads": 128, "topk": 2048, "rows": 32768},
        # a ragged chunk of a longer prompt on one of eight ranks that share the heads out
        {"name": "attend_1999_tokens_16_heads", "kind": "attend", "tokens": 1999, "heads": 16, "topk": 2048, "rows": 4801},
        # prefill of 4096 tokens with all heads, causal from the first token: the headline workload
        {"name": "attend_4096_tokens", "kind": "attend", "tokens": 4096, "heads": 128, "topk": 2048, "rows": 4096},
        # a decode step of a nearly idle server
        {"name": "step_3_sequences", "kind": "step", "batch": 3, "n_q": 1, "heads": 128, "topk": 2048, "len_lo": 3000, "len_hi": 20000},
        # a decode step under load, two tokens per sequence (one of them speculative)
        {"name": "step_64_sequences", "kind": "step", "batch": 64, "n_q": 2, "heads": 128, "topk": 2048, "len_lo": 8192, "len_hi": 65536},
        # the latent rows of a large prefill batch go to the cache
        {"name": "fill_262144_rows", "kind": "fill", "new_rows": 262144},
        # index lists of a 4096-token chunk over a 32768-token context
        {"name": "select_4096x32768", "kind": "select", "tokens": 4096, "rows": 32768, "topk": 2048},
        # eight ranks hold an eighth of the context each
        {"name": "merge_8_parts", "kind": "merge", "parts": 8, "tokens": 512, "heads": 128, "fp32": False},
        # a row-parallel projection in decode, and the same weight in prefill
        {"name": "matmul_50_rows", "kind": "matmul", "m": 50, "n": 7168, "k": 2304},
        {"name": "matmul_8192_rows", "kind": "matmul", "m": 8192, "n": 7168, "k": 2304},
        # FP8 projection with a linear layer's [N, K] weight in decode, and with a [K, N] weight in prefill
        {"name": "matmul8_64_rows", "kind": "matmul8", "m": 64, "n": 8192, "k": 3584, "nk": True},
        {"name": "matmul8_4096_rows", "kind": "matmul8", "m": 4096, "n": 8192, "k": 28672, "nk": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attend", "attend", "attend", "step", "fill", "select", "merge", "matmul", "matmul", "matmul8", "matmul8"])
    if kind == "attend":
        tokens = _log(rng, 1, 4096)
        topk = rng.choice([2048, 2048, 1024, 512, 256, rng.randint(65, 2047)])
        return {"kind": kind, "tokens": tokens, "heads": rng.choice([128, 128, 64, 32, 16]), "topk": topk,
                "rows": max(tokens, topk) + _log(rng, 1, 60000 if tokens < 256 else 4096)}
    if kind == "step":
        lo = _log(rng, 2048, 16384)
        return {"kind": kind, "batch": _log(rng, 1, 64), "n_q": rng.choice([1, 1, 2]), "heads": rng.choice([128, 128, 64, 16]),
                "topk": rng.choice([2048, 2048, 1024, 512]), "len_lo": lo, "len_hi": lo + _log(rng, 1000, 49152)}
    if kind == "fill":
        return {"kind": kind, "new_rows": _log(rng, 64, 262144)}
    if kind == "select":
        return {"kind": kind, "tokens": _log(rng, 1, 4096), "rows": _log(rng, 3000, 32768), "topk": rng.choice([2048, 2048, 1024, 512])}
    if kind == "merge":
        return {"kind": kind, "parts": rng.choice([2, 4, 8]), "tokens": _log(rng, 1, 512), "heads": rng.choice([128, 64, 16]),
                "fp32": rng.random() < 0.3}
    if kind == "matmul":
        return {"kind": kind, "m": _log(rng, 1, 8192), "n": 8 * rng.randint(64, 896), "k": 8 * rng.randint(64, 288)}
    k = 128 * rng.randint(8, 56) if rng.random() < 0.7 else 128 * rng.randint(57, 224)
    return {"kind": kind, "m": _log(rng, 1, 4096), "n": 128 * rng.randint(8, 64), "k": k, "nk": rng.random() < 0.6}


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV)


def _visible(c):
    """How many rows of the context each token of an `attend` or `select` case sees."""
    first = c["rows"] - c["tokens"]
    return [first + t + 1 for t in range(c["tokens"])]


def _choose(g, seen, rows, topk):
    """[tokens, topk] int32: per token min(topk, seen) distinct positions below its `seen`, ascending, -1 behind."""
    out = torch.full((len(seen), topk), -1, dtype=torch.int32, device=DEV)
    lens = torch.tensor(seen, device=DEV)
    pos = torch.arange(rows, device=DEV)
    for a in range(0, len(seen), 1024):
        n = lens[a:a + 1024, None]
        keys = torch.rand(n.shape[0], rows, generator=g, device=DEV)
        keys.masked_fill_(pos[None, :] >= n, -1.0)
        got = keys.topk(min(topk, rows), dim=1)
        at = torch.where(got.values >= 0, got.indices, rows).sort(dim=1).values
        out[a:a + 1024, :at.shape[1]] = torch.where(at < rows, at, -1).to(torch.int32)
    return out


def _quantise(x, block_r, block_c):
    """fp32 [R, C] -> e4m3 and the fp32 scales of its blocks."""
    r, c = x.shape
    xb = x.view(r // block_r, block_r, c // block_c, block_c)
    scale = xb.abs().amax(dim=(1, 3)).clamp(min=1e-12) / 448.0
    return (xb / scale[:, None, :, None]).to(torch.float8_e4m3fn).view(r, c), scale


def prepare(case, seed):
    g, c = _gen(seed), case
    kind = c["kind"]
    if kind == "attend":
        return {"kind": kind, "q": _randn(g, c["tokens"], c["heads"], D_QK).bfloat16(), "kv": _randn(g, c["rows"], D_QK).bfloat16(),
                "indices": _choose(g, _visible(c), c["rows"], c["topk"])}
    if kind == "step":
        batch, n_q = c["batch"], c["n_q"]
        # lengths spread over [len_lo, len_hi], the same ones for every seed so that the shapes are the case's own
        held = [c["len_lo"] + int((c["len_hi"] - c["len_lo"]) * ((b + 1) * 0.618034 % 1.0)) for b in range(batch)]
        lens = torch.tensor(held, device=DEV)
        pages = [-(-n // PAGE) for n in held]
        order = torch.randperm(sum(pages), generator=g, device=DEV).to(torch.int32)
        table = torch.zeros(batch, max(pages), dtype=torch.int32, device=DEV)
        at = 0
        for b, n in enumerate(pages):
            table[b, :n] = order[at:at + n]
            at += n
        cache = torch.empty(at, PAGE, D_QK, dtype=torch.float8_e4m3fn, device=DEV)
        scale = torch.empty(at, device=DEV)
        for a in range(0, at, 4096):
            x = _randn(g, min(4096, at - a), PAGE * D_QK)
            q8, s = _quantise(x, 1, PAGE * D_QK)
            cache[a:a + 4096], scale[a:a + 4096] = q8.view(-1, PAGE, D_QK), s[:, 0]
        # the n_q new tokens of a sequence are its last positions; token j sees the positions up to its own
        where = (lens[:, None] - n_q + torch.arange(n_q, device=DEV)[None, :])
        slots = table.gather(1, where // PAGE) * PAGE + (where % PAGE).to(torch.int32)
        return {"kind": kind, "rows": _randn(g, batch * n_q, D_QK).bfloat16(), "slots": slots.reshape(-1).to(torch.int32).contiguous(),
                "cache": cache.view(torch.uint8), "scale": scale, "table": table, "lens": lens.to(torch.int32),
                "scores": _randn(g, batch * n_q, max(pages) * PAGE), "seen": (where + 1).reshape(-1).to(torch.int32).contiguous(),
                "topk": c["topk"], "q": _randn(g, batch, n_q, c["heads"], D_QK).bfloat16()}
    if kind == "fill":
        pages = -(-c["new_rows"] // PAGE)
        order = torch.randperm(pages, generator=g, device=DEV)
        n = torch.arange(c["new_rows"], device=DEV)
        return {"kind": kind, "rows": _randn(g, c["new_rows"], D_QK).bfloat16(), "slots": (order[n // PAGE] * PAGE + n % PAGE).to(torch.int32),
                "cache": torch.zeros(pages, PAGE, D_QK, dtype=torch.uint8, device=DEV), "scale": torch.zeros(pages, device=DEV)}
    if kind == "select":
        seen = [min(c["rows"], max(1, n)) for n in _visible(c)] if c["rows"] > c["tokens"] else [c["rows"]] * c["tokens"]
        return {"kind": kind, "scores": _randn(g, c["tokens"], c["rows"]), "seen": torch.tensor(seen, dtype=torch.int32, device=DEV), "topk": c["topk"]}
    if kind == "merge":
        part = _randn(g, c["parts"], c["tokens"], c["heads"], D_V)
        return {"kind": kind, "out": part if c["fp32"] else part.bfloat16(), "lse": _randn(g, c["parts"], c["tokens"], c["heads"]) + 7.0}
    if kind == "matmul":
        s = c["k"] ** -0.5
        return {"kind": kind, "a": (_randn(g, c["m"], c["k"]) * s).bfloat16(), "b": (_randn(g, c["k"], c["n"]) * s).bfloat16()}
    a, a_scale = _quantise(_randn(g, c["m"], c["k"]), 1, 128)
    w, w_scale = _quantise(_randn(g, c["n"], c["k"]) if c["nk"] else _randn(g, c["k"], c["n"]), 128, 128)
    return {"kind": kind, "a": a, "a_scale": a_scale, "b": w.t() if c["nk"] else w, "b_scale": w_scale.t().contiguous() if c["nk"] else w_scale}


def run(s):
    kind = s["kind"]
    if kind == "attend":
        return ft.sparse_mla_fwd(s["q"], s["kv"], s["indices"], SM_SCALE)
    if kind == "step":
        ft.kv_cache_write_fp8(s["rows"], s["slots"], s["cache"], s["scale"], PAGE)
        chosen = ft.topk_indices(s["scores"], s["topk"], s["seen"])
        b, n_q = s["q"].shape[:2]
        out, lse = ft.sparse_mla_fwd_paged(s["q"], s["cache"], s["scale"], s["table"], s["lens"], chosen.view(b, n_q, -1), SM_SCALE)
        return chosen, out, lse, s["cache"], s["scale"]
    if kind == "fill":
        ft.kv_cache_write_fp8(s["rows"], s["slots"], s["cache"], s["scale"], PAGE)
        return s["cache"], s["scale"]
    if kind == "select":
        return ft.topk_indices(s["scores"], s["topk"], s["seen"])
    if kind == "merge":
        return ft.sparse_mla_merge(s["out"], s["lse"])
    if kind == "matmul":
        return ft.matmul(s["a"], s["b"])
    return ft.matmul_fp8_blockscaled(s["a"], s["a_scale"], s["b"], s["b_scale"])


def work(case):
    c, kind = case, case["kind"]
    if kind == "attend":
        chosen = sum(min(n, c["topk"]) for n in _visible(c))
        rows = min(c["rows"], chosen)
        return {"bytes": c["tokens"] * c["heads"] * (2 * D_QK + 2 * D_V + 4) + 2 * D_QK * rows + 4 * c["tokens"] * c["topk"],
                "flops": 2 * (D_QK + D_V) * c["heads"] * chosen}
    if kind == "step":
        tokens = c["batch"] * c["n_q"]
        seen = (c["len_lo"] + c["len_hi"]) / 2
        chosen = min(c["topk"], c["len_lo"])
        return {"bytes": tokens * (D_QK * (2 + 1) + 4 * seen + 8 * c["topk"] + D_QK * chosen + c["heads"] * (2 * D_QK + 2 * D_V + 4)),
                "flops": 2 * (D_QK + D_V) * c["heads"] * chosen * tokens}
    if kind == "fill":
        return {"bytes": c["new_rows"] * (2 * D_QK + 4 + D_QK) + 4 * -(-c["new_rows"] // PAGE), "flops": 0}
    if kind == "select":
        seen = sum(_visible(c)) if c["rows"] > c["tokens"] else c["rows"] * c["tokens"]
        return {"bytes": 4 * seen + 4 * c["tokens"] * c["topk"], "flops": 0}
    if kind == "merge":
        return {"bytes": c["tokens"] * c["heads"] * (c["parts"] * (D_V * (4 if c["fp32"] else 2) + 4) + D_V * 2 + 4), "flops": 0}
    size = 2 if kind == "matmul" else 1
    scales = 0 if kind == "matmul" else 4 * (c["m"] * c["k"] // 128 + c["n"] * c["k"] // (128 * 128))
    return {"bytes": size * (c["m"] + c["n"]) * c["k"] + 2 * c["m"] * c["n"] + scales, "flops": 2 * c["m"] * c["n"] * c["k"]}


def tolerance(case):
    # Measured against the same arithmetic in 64 bits (relative 2-norm, largest difference), then about four times
    # that: attend 0.0021 and 0.012, step 0.0040 and 0.037, merge and the matrix products 0.0017 and 0.0039 (bf16 results).
    kind = case["kind"]
    if kind in ("fill", "select"):
        return "exact"                           # bytes, scales and positions have one right answer
    if kind == "attend":
        return {"rel": 8e-3, "max": 0.05}
    if kind == "step":
        return {"rel": 1.2e-2, "max": 0.12}
    return {"rel": 7e-3, "max": 0.016}
