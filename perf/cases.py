"""Performance cases of the quantize -> pack -> attend path: what a program that uses this package has it do.

Every case goes through the public entry points of `turboquant_b200`.  Kinds:

  kv_attend   QuantizedKVCache on host arrays: scores of one query over all keys, softmax, weighted values
  generate    PqoCache, one request: new sequence, prompt stored, then a few decode steps over all layers
  decode      PqoCache, one decode step of a running batch: append + attention, layer after layer
  tq_decode   TqCache, the same with the sign-sketch correction inside the attention
  chunk       causal attention of a prefill chunk over packed keys / values that are stored already
  prompt      PqoCache, a prompt taken in by chunks: quantize, store, attend
  tq_prompt   TqCache, a prompt taken in by chunks (dequantized cache and logit bias handed back), one decode step
  block       block-32 format: quantize rows and dequantize them again
  whole       whole-vector format: quantize rows and dequantize them again
  qjl_list    whole-vector format with sign sketch: quantize a list of keys, score a query over it, weigh values

Shapes are those of the benchmark and the tests (head_dim 128, 8 KV heads, groups of 1 to 8 query heads), and odd
sizes between them.  Keys and values are normal with a spread per channel: 4-bit caches log-normal(0, 0.5), 3-bit
caches 3 channels of 128 scaled by 8.
"""
import math

import numpy as np
import torch

import turboquant_b200 as tq

D = 128                      # head_dim of the cache cases
SCALE = 1.0 / math.sqrt(D)
QJL_SEED = 42
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def listed():
    return [
        # the smallest calls: a single head's host-side cache of 1,024 entries
        dict(name="kv_attend_1k", kind="kv_attend", bits=3, dim=128, n=1024),
        # a short request on a small model, batch 1: launches and host work per layer count
        dict(name="generate_b1_1k_3bit", kind="generate", bits=3, dtype="bf16", batch=1, hq=16, hkv=8, ctx=1024, steps=16, layers=28),
        # serving a full batch at 8K context, 4-bit: the largest ordinary decode step
        dict(name="decode_b64_8k_4bit", kind="decode", bits=4, dtype="bf16", batch=64, hq=32, hkv=8, ctx=8192, layers=8),
        # serving a middling batch at an odd context, 3-bit
        dict(name="decode_b24_5001_3bit", kind="decode", bits=3, dtype="bf16", batch=24, hq=32, hkv=8, ctx=5001, layers=16),
        # one long document, 8 query heads per KV head, 3-bit
        dict(name="decode_b1_128k_3bit", kind="decode", bits=3, dtype="bf16", batch=1, hq=64, hkv=8, ctx=131072, layers=8),
        # decode with the sketch-corrected scores
        dict(name="tq_decode_b16_4001", kind="tq_decode", bits=3, dtype="bf16", batch=16, hq=32, hkv=8, ctx=4001, layers=8),
        # a prefill chunk of 512 tokens that ends at 8,192
        dict(name="chunk_512_at_8k_4bit", kind="chunk", bits=4, dtype="bf16", hq=32, hkv=8, q_len=512, past=7680),
        # a prompt of odd length taken in by chunks of 1,024
        dict(name="prompt_1999_4bit", kind="prompt", bits=4, dtype="bf16", batch=1, hq=32, hkv=8, tokens=1999, chunk=1024, layers=4),
        # the sketch cache taking in a batch of prompts
        dict(name="tq_prompt_b8_384", kind="tq_prompt", bits=3, dtype="bf16", batch=8, hq=32, hkv=8, tokens=384, chunk=96, layers=2),
        # bulk quantize / dequantize of cache rows: encode and decode
        dict(name="block_1m_4bit", kind="block", bits=4, dtype="bf16", n=1048576),
        # the same for the whole-vector format
        dict(name="whole_512k_3bit", kind="whole", bits=3, dim=128, n=524288),
        # a list of sketched keys: insertion, then one query over it
        dict(name="qjl_list_64k_4bit", kind="qjl_list", bits=4, dim=128, n=65536),
    ]


def _log(rng, lo, hi):
    """An odd or even size between lo and hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["kv_attend", "generate", "decode", "decode", "tq_decode", "chunk", "prompt", "tq_prompt", "block", "whole", "qjl_list"])
    c = dict(kind=kind)
    hkv = 8
    group = rng.choice([1, 2, 4, 8])
    bits = rng.choice([3, 4])
    dtype = rng.choice(["bf16", "bf16", "f16", "f32"])
    if kind == "kv_attend":
        c.update(bits=bits, dim=rng.choice([64, 128, 256]), n=_log(rng, 64, 65536))
    elif kind == "generate":
        c.update(bits=bits, dtype=dtype, batch=rng.choice([1, 1, 2, 3]), hq=hkv * group, hkv=hkv, ctx=_log(rng, 100, 4096),
                 steps=rng.randint(4, 16), layers=rng.randint(8, 28))
    elif kind == "decode":
        # at most 64 x 8192 tokens a layer
        ctx = _log(rng, 1024, 131072)
        c.update(bits=bits, dtype=dtype, batch=_log(rng, 1, max(1, min(64, 64 * 8192 // ctx))), hq=hkv * group, hkv=hkv, ctx=ctx, layers=8)
    elif kind == "tq_decode":
        ctx = _log(rng, 1024, 32768)
        c.update(bits=3, dtype=dtype, batch=_log(rng, 1, max(1, min(16, 16 * 4096 // ctx))), hq=hkv * group, hkv=hkv, ctx=ctx, layers=8)
    elif kind == "chunk":
        c.update(bits=bits, dtype=dtype, hq=hkv * group, hkv=hkv, q_len=_log(rng, 16, 2048), past=rng.choice([0, _log(rng, 128, 16384)]))
    elif kind == "prompt":
        c.update(bits=bits, dtype=dtype, batch=1, hq=hkv * group, hkv=hkv, tokens=_log(rng, 100, 4096), chunk=rng.choice([512, 1024, 2048]),
                 layers=rng.randint(2, 6))
    elif kind == "tq_prompt":
        c.update(bits=3, dtype=dtype, batch=rng.randint(1, 8), hq=hkv * min(group, 4), hkv=hkv, tokens=_log(rng, 60, 600),
                 chunk=rng.choice([48, 64, 96]), layers=2)
    elif kind == "block":
        c.update(bits=bits, dtype=dtype, n=_log(rng, 1000, 2097152))
    elif kind == "whole":
        c.update(bits=rng.choice([2, 3, 4]), dim=rng.choice([64, 128, 256]), n=_log(rng, 1000, 1048576))
    else:
        c.update(bits=bits, dim=rng.choice([64, 128]), n=_log(rng, 1000, 131072))
    return c


# ---- inputs -------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _spread(bits, g):
    """Per-channel spread of a layer's keys or values."""
    if bits == 4:
        return torch.exp(torch.randn(D, generator=g, device="cuda") * 0.5)
    s = torch.ones(D, device="cuda")
    s[torch.randperm(D, generator=g, device="cuda")[:3]] = 8.0
    return s


def _kv(shape, spread, g, dtype):
    return (torch.randn(shape, generator=g, device="cuda") * spread).to(dtype)


def _rows(case, tokens, g, spreads):
    """k, v of `tokens` tokens and q of as many, as a layer's projections hand them over."""
    dt, b = DTYPES[case["dtype"]], case.get("batch", 1)
    k = _kv((b, case["hkv"], tokens, D), spreads[0], g, dt)
    v = _kv((b, case["hkv"], tokens, D), spreads[1], g, dt)
    # queries shaped so that the logits have a spread of about 2 whatever the keys' channel spread
    q = torch.randn((b, case["hq"], tokens, D), generator=g, device="cuda") * (2.0 / float(spreads[0].square().mean().sqrt()))
    return k, v, q.to(dt)


def _cache_config(case, sketch=False):
    return tq.CacheConfig(bits=case["bits"], head_dim=D, num_kv_heads=case["hkv"], num_layers=case["layers"], batch=case["batch"],
                          outlier_blocks=0 if sketch else tq.ALL_BLOCKS)


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    s = dict(case=case)
    if kind == "kv_attend":
        rng = np.random.default_rng(seed)
        cfg = tq.TurboQuantConfig(case["bits"], case["dim"]).with_seed(QJL_SEED)
        s["cache"] = tq.QuantizedKVCache(cfg, 1, QJL_SEED)
        shape = (case["n"], case["dim"])
        s["cache"].push_batch(0, rng.standard_normal(shape, dtype=np.float32), rng.standard_normal(shape, dtype=np.float32))
        s["q"] = (rng.standard_normal(case["dim"], dtype=np.float32) / np.float32(math.sqrt(case["dim"]))).astype(np.float32)
    elif kind in ("generate", "decode", "tq_decode", "prompt", "tq_prompt"):
        sketch = kind.startswith("tq_")
        s["cache"] = (tq.TqCache if sketch else tq.PqoCache)(_cache_config(case, sketch))
        s["att"] = tq.AttendConfig(SCALE, case["hq"] // case["hkv"])
        layers = []
        for layer in range(case["layers"]):
            spreads = (_spread(case["bits"], g), _spread(case["bits"], g))
            if kind == "generate":
                k, v, _ = _rows(case, case["ctx"], g, spreads)
                layers.append((k, v, [_rows(case, 1, g, spreads) for _ in range(case["steps"])]))
            elif kind in ("decode", "tq_decode"):
                k, v, q = _rows(case, case["ctx"], g, spreads)
                if sketch:
                    s["cache"].prefill(layer, k, v, q[:, :, -1:].contiguous())
                else:
                    s["cache"].prefill(layer, k, v)
                del k, v, q
                layers.append(_rows(case, 1, g, spreads))
            else:
                k, v, q = _rows(case, case["tokens"] + (1 if sketch else 0), g, spreads)
                layers.append([tuple(t[:, :, a:b].contiguous() for t in (k, v, q)) for a, b in _pieces(case)])
        s["layers"] = layers
    elif kind == "chunk":
        spreads = (_spread(case["bits"], g), _spread(case["bits"], g))
        n = case["past"] + case["q_len"]
        k, v, _ = _rows(case, n, g, spreads)
        s["kv"] = []
        for t in (k, v):
            idx, sc = tq.block_quantize(t.reshape(-1, D), case["bits"])
            s["kv"] += [idx.view(case["hkv"], n, -1), sc.view(case["hkv"], n, -1)]
        q = torch.randn((case["q_len"], case["hq"], D), generator=g, device="cuda") * (2.0 / float(spreads[0].square().mean().sqrt()))
        s["q"] = q.to(DTYPES[case["dtype"]])
    elif kind == "block":
        s["x"] = _kv((case["n"], D), _spread(case["bits"], g), g, DTYPES[case["dtype"]])
    elif kind == "whole":
        s["cfg"] = tq.TurboQuantConfig(case["bits"], case["dim"]).with_seed(QJL_SEED)
        s["x"] = torch.randn((case["n"], case["dim"]), generator=g, device="cuda")
    else:
        s["cfg"] = tq.TurboQuantConfig(case["bits"], case["dim"]).with_seed(QJL_SEED)
        s["x"] = torch.randn((case["n"], case["dim"]), generator=g, device="cuda")
        s["q"] = torch.randn((case["dim"],), generator=g, device="cuda") / math.sqrt(case["dim"])
        w = torch.rand((case["n"],), generator=g, device="cuda")
        s["w"] = w / w.sum()
    return s


def _pieces(case):
    """Token ranges of a prompt's chunks; the sketch cache's prompt is followed by the token of one decode step."""
    n, c = case["tokens"], case["chunk"]
    got = [(a, min(a + c, n)) for a in range(0, n, c)]
    return got + [(n, n + 1)] if case["kind"] == "tq_prompt" else got


# ---- one pass -----------------------------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    return _RUN[case["kind"]](s, case)


def _run_kv_attend(s, case):
    scores = s["cache"].attention_scores(0, s["q"])
    w = np.exp(scores - scores.max())
    w /= w.sum()
    return scores, s["cache"].weighted_values(0, w)


def _run_generate(s, case):
    cache, att, layers = s["cache"], s["att"], s["layers"]
    cache.reset()
    for layer, (k, v, _) in enumerate(layers):
        cache.prefill(layer, k, v)
    for step in range(case["steps"]):
        outs = []
        for layer, (_, _, rows) in enumerate(layers):
            k, v, q = rows[step]
            outs.append(cache.decode(layer, k, v, q, att).fused)
    return outs


def _run_decode(s, case):
    cache, att = s["cache"], s["att"]
    return [cache.decode(layer, k, v, q, att).fused for layer, (k, v, q) in enumerate(s["layers"])]


def _run_tq_decode(s, case):
    cache, att = s["cache"], s["att"]
    return [cache.decode_fused(layer, k, v, q, att).fused for layer, (k, v, q) in enumerate(s["layers"])]


def _run_chunk(s, case):
    ki, ks, vi, vs = s["kv"]
    return tq.chunk_attention(s["q"], ki, ks, vi, vs, case["past"] + case["q_len"], case["bits"], SCALE)


def _run_prompt(s, case):
    cache, att, layers = s["cache"], s["att"], s["layers"]
    cache.reset()
    outs = []
    for piece in range(len(layers[0])):
        for layer, rows in enumerate(layers):
            k, v, q = rows[piece]
            outs.append(cache.prefill_attend(layer, k, v, q, att))
    return outs


def _run_tq_prompt(s, case):
    cache, layers = s["cache"], s["layers"]
    cache.reset()
    last = len(layers[0]) - 1
    outs = []
    for piece in range(last):
        for layer, rows in enumerate(layers):
            k, v, q = rows[piece]
            r = cache.prefill(layer, k, v, q)
            outs.append(r.logit_bias)
    for layer, rows in enumerate(layers):
        k, v, q = rows[last]
        r = cache.decode(layer, k, v, q).dequantized
        outs += [r.k, r.v, r.logit_bias]
    return outs


def _run_block(s, case):
    idx, sc = tq.block_quantize(s["x"], case["bits"])
    return idx, sc, tq.block_dequantize(idx, sc, case["bits"], D, dtype=s["x"].dtype)


def _run_whole(s, case):
    packed, scales = tq.quantize_batch(s["cfg"], s["x"])
    return packed, scales, tq.dequantize_batch(s["cfg"], packed, scales)


def _run_qjl_list(s, case):
    cfg = s["cfg"]
    packed, scales, signs, rnorms = tq.qjl_quantize_batch(cfg, s["x"], QJL_SEED)
    rq = tq.query_projections(s["q"], case["dim"], QJL_SEED)
    scores = tq.qjl_attention_scores(cfg, s["q"], rq, packed, scales, signs, rnorms)
    return packed, scales, signs, rnorms, scores, tq.weighted_values(cfg, s["w"], packed, scales)


_RUN = {"kv_attend": _run_kv_attend, "generate": _run_generate, "decode": _run_decode, "tq_decode": _run_tq_decode, "chunk": _run_chunk,
        "prompt": _run_prompt, "tq_prompt": _run_tq_prompt, "block": _run_block, "whole": _run_whole, "qjl_list": _run_qjl_list}


# ---- what a pass cannot do without --------------------------------------------------------------------------------
def _esize(case):
    return 4 if case.get("dtype", "f32") == "f32" else 2


def _row_bytes(bits, sketch=False):
    """Stored bytes of one token of one KV head, K and V."""
    return 2 * (D * bits // 8 + 2 * (D // 32)) + (D // 8 + 2 if sketch else 0)


def work(case):
    kind, e = case["kind"], _esize(case)
    if kind == "kv_attend":
        n, d, polar = case["n"], case["dim"], case["dim"] * (case["bits"] - 1) // 8
        return {"bytes": n * (2 * (polar + 2) + d // 8 + 2 + 8) + 8 * d, "flops": n * d * 6}
    if kind in ("decode", "tq_decode", "generate"):
        b, hq, hkv, ctx = case["batch"], case["hq"], case["hkv"], case["ctx"]
        steps = case.get("steps", 1)
        seen = sum(ctx + 1 + i for i in range(steps))
        row = _row_bytes(case["bits"], kind == "tq_decode")
        by = b * hkv * seen * row + steps * b * (2 * hq + 2 * hkv) * D * e
        if kind == "generate":
            by += b * hkv * ctx * (2 * D * e + row)
        return {"bytes": case["layers"] * by, "flops": case["layers"] * b * hq * seen * D * (6 if kind == "tq_decode" else 4)}
    if kind == "chunk":
        n, past = case["q_len"], case["past"]
        seen = n * past + n * (n + 1) // 2
        return {"bytes": case["hkv"] * (past + n) * _row_bytes(case["bits"]) + 2 * n * case["hq"] * D * e, "flops": 4 * case["hq"] * D * seen}
    if kind == "prompt":
        n = case["tokens"]
        by = n * (2 * case["hkv"] + 2 * case["hq"]) * D * e + n * case["hkv"] * _row_bytes(case["bits"])
        return {"bytes": case["layers"] * case["batch"] * by, "flops": case["layers"] * case["batch"] * 4 * case["hq"] * D * n * (n + 1) // 2}
    if kind == "tq_prompt":
        hq, hkv, by, fl = case["hq"], case["hkv"], 0, 0
        for i, (a, b) in enumerate(_pieces(case)):
            rows = (b - a) * hkv
            by += rows * (2 * D * e + _row_bytes(case["bits"], True)) + (b - a) * hq * (D + b) * e   # in, stored, q, bias
            by += (2 * hkv * b * D * e + hkv * a * _row_bytes(case["bits"], True)) if i else 0       # dequantized cache handed back
            fl += 2 * D * (b - a) * hq * b + 2 * D * D * (rows + (b - a) * hq)                       # bias, sketch, projections
        return {"bytes": case["layers"] * case["batch"] * by, "flops": case["layers"] * case["batch"] * fl}
    if kind == "block":
        return {"bytes": case["n"] * (2 * D * e + _row_bytes(case["bits"])), "flops": case["n"] * D * 10}
    n, d = case["n"], case["dim"]
    if kind == "whole":
        return {"bytes": n * (8 * d + 2 * (d * case["bits"] // 8 + 2)), "flops": n * d * 4 * int(math.log2(d))}
    polar = d * (case["bits"] - 1) // 8
    return {"bytes": n * (4 * d + 2 * (polar + d // 8 + 4) + polar + 2 + 8), "flops": n * (2 * d * d + 6 * d)}


def tolerance(case):
    """About four times what each path shows against itself in 64 bits over the same stored codes."""
    kind, dt = case["kind"], case.get("dtype", "f32")
    if kind in ("block", "whole"):
        return "exact"       # every code, scale and dequantized value is defined bit by bit
    if kind in ("kv_attend", "qjl_list"):
        return {"rel": 1e-5, "max": 1e-4}      # f32 sums; seen 2e-7 (codes, scales and signs: exact)
    if dt == "bf16":         # the outputs' own rounding; seen 1.7e-3
        r = {"rel": 7e-3, "max": 2e-2}
    elif dt == "f16":        # seen 2.3e-4
        r = {"rel": 1e-3, "max": 4e-3}
    elif case["bits"] == 3 and kind in ("decode", "generate"):
        r = {"rel": 4e-4, "max": 3e-3}         # 3-bit centroids held as f16; seen 1e-4
    else:                    # f32 sums; seen 3e-6
        r = {"rel": 1.2e-5, "max": 1.2e-4}
    if kind in ("chunk", "prompt"):            # f16 operands on the tensor cores; seen 1.1e-3 (bf16 outputs: 2e-3), max 0.09
        r = {"rel": 8e-3 if dt == "bf16" else 4.5e-3, "max": 0.35}
    return r
