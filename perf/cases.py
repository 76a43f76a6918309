"""The work that a user of this package has it do, as cases that can be timed and compared.

The package packs vectors (``TurboQuantMSE``, ``TurboQuantProd``), scores queries against packed keys, keeps a packed
key / value cache for decoding and searches packed key sets.  The cases take these through the public classes, at the
sizes of the repository's own configurations, tests and benchmark, from one token per sequence to 16,777,216 keys:

  append     one decode step's keys and values go into a ``PackedKVCache`` (latency and launches count)
  prefill    a whole prompt's keys and values go into a ``PackedKVCache``
  attend     one decode step's attention over a filled ``PackedKVCache``
  mse        ``TurboQuantMSE``: quantize, then dequantize
  prod       ``TurboQuantProd``: quantize keys
  sweep      ``TurboQuantProd``: quantize, dequantize and 16-query scores (the dimension / bit-width sweep)
  harness    the validation harness's calls on NumPy arrays, a few hundred vectors, one query at a time
  score_one  ``attention_score``: one query against every key
  scores     ``attention_scores``: the whole score matrix of a batch of queries
  search     ``ShardedKeyIndex.search``: the best keys of every query, no matrix

Quantizers are built once per geometry and kept, as a program keeps them; inputs are made from the seed alone.
"""
import math

import numpy as np
import torch

import project_tensor_b200 as tg
from project_tensor_b200.sharded import ShardedKeyIndex

#: seed of every quantizer's rotation and projection (the configurations' own)
QUANTIZER_SEED = 2026
#: channels per key head that are ten times as large as the others in key / value caches
OUTLIER_CHANNELS = 4

_DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16, "float16": torch.float16}
_quantizers = {}


def _quantizer(kind, d, bits):
    key = (kind, d, bits)
    if key not in _quantizers:
        make = {"mse": tg.TurboQuantMSE, "prod": tg.TurboQuantProd}[kind]
        _quantizers[key] = make(d, bits, seed=QUANTIZER_SEED)
    return _quantizers[key]


# ------------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------------
def listed():
    return [
        # decode, 8 sequences x 8 key heads: the new token's keys and values, every step of every layer
        {"name": "append_64x1", "op": "append", "groups": 64, "d": 128, "bits": 4, "vbits": 4, "dtype": "float32"},
        # the reference's validation harness: 256 NumPy vectors, 32 queries scored one call at a time
        {"name": "harness_256_numpy", "op": "harness", "n": 256, "queries": 32, "d": 64, "bits": 4},
        # decode over a short context, one query per key head, small heads
        {"name": "attend_32x1x1531_d64", "op": "attend", "groups": 32, "queries": 1, "keys": 1531, "d": 64, "bits": 4,
         "vbits": 3, "dtype": "float32"},
        # decode over a long context, grouped queries 4:1 (the KV-cache configuration)
        {"name": "attend_64x4x32768", "op": "attend", "groups": 64, "queries": 4, "keys": 32768, "d": 128, "bits": 4,
         "vbits": 4, "dtype": "float32"},
        # prefill of the same cache by a model that computes in bf16
        {"name": "prefill_64x4096_bf16", "op": "prefill", "groups": 64, "tokens": 4096, "d": 128, "bits": 3, "vbits": 4,
         "dtype": "bfloat16"},
        # the first configuration: pack and restore 65,536 vectors
        {"name": "mse_65536", "op": "mse", "n": 65536, "d": 128, "bits": 4},
        # the second configuration: pack 1,048,576 keys, then 32 queries against all of them
        {"name": "prod_1048576", "op": "prod", "n": 1048576, "d": 128, "bits": 4},
        {"name": "scores_32x1048576", "op": "scores", "n": 1048576, "queries": 32, "d": 128, "bits": 4},
        # the sweep at its largest dimension, a ragged count
        {"name": "sweep_524309_d256", "op": "sweep", "n": 524309, "d": 256, "bits": 4},
        # the sweep at a head size that is no power of two, at the harness's largest bit width
        {"name": "sweep_50021_d96_b6", "op": "sweep", "n": 50021, "d": 96, "bits": 6},
        # the reference's own scoring call, a ragged count
        {"name": "score_one_262147", "op": "score_one", "n": 262147, "d": 128, "bits": 4},
        # retrieval: one GPU's share of 134,217,728 keys over 8
        {"name": "search_64x16777216", "op": "search", "n": 16777216, "queries": 64, "topk": 100, "d": 128, "bits": 4},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["append", "prefill", "attend", "attend", "mse", "prod", "sweep", "harness", "score_one", "scores",
                     "search"])
    case = {"op": op}
    if op in ("append", "prefill", "attend"):
        case["d"] = rng.choice([64, 128])
        case["bits"], case["vbits"] = rng.choice([2, 3, 4]), rng.choice([2, 3, 4])
        case["dtype"] = rng.choice(["float32", "bfloat16", "float16"])
        case["groups"] = _log_uniform(rng, 4, 256)
        if op == "prefill":
            case["tokens"] = _log_uniform(rng, 32, min(16384, (1 << 19) // case["groups"]))
        if op == "attend":
            case["queries"] = rng.choice([1, 2, 4, 8])
            case["keys"] = _log_uniform(rng, 128, min(131072, (1 << 22) // case["groups"]))
        return case
    if op == "harness":
        case["d"], case["bits"] = rng.choice([64, 128, 256]), rng.choice([2, 4, 6])
        case["n"], case["queries"] = _log_uniform(rng, 64, 2048), rng.randint(4, 32)
        return case
    if op in ("mse", "prod", "sweep"):
        case["d"], case["bits"] = rng.choice([64, 96, 128, 128, 256]), rng.choice([1, 2, 3, 4, 4, 6])
        common = case["d"] != 96 and case["bits"] <= 4
        case["n"] = _log_uniform(rng, 1000, (1 << 27) // case["d"] if common else 1 << 16)
        return case
    case["d"], case["bits"] = rng.choice([64, 128, 128, 256]), rng.choice([2, 3, 4])
    if op == "score_one":
        case["n"] = _log_uniform(rng, 1000, 1 << 22)
    elif op == "scores":
        case["queries"] = _log_uniform(rng, 2, 64)
        case["n"] = _log_uniform(rng, 1000, 1 << 20)
    else:
        case["queries"], case["topk"] = _log_uniform(rng, 1, 64), rng.choice([10, 100])
        case["n"] = _log_uniform(rng, 65536, (1 << 30) // case["d"])
    return case


# ------------------------------------------------------------------------------------------------
# what the program has in hand before the call
# ------------------------------------------------------------------------------------------------
def _normal(shape, gen, scale=1.0):
    x = torch.randn(shape, device="cuda", generator=gen)
    return x if scale == 1.0 else x.mul_(scale)


def _cache_rows(groups, tokens, d, gen):
    """Keys (or values) of a cache: N(0, 1) with a few large channels per head, fixed over its tokens."""
    x = _normal((groups, tokens, d), gen)
    loud = torch.rand((groups, d), device="cuda", generator=gen).topk(OUTLIER_CHANNELS, dim=1).indices
    factor = torch.ones((groups, d), device="cuda").scatter_(1, loud, 10.0)
    return x.mul_(factor[:, None, :])


def _key_index(quant, n, d, gen):
    """An index of n packed keys, filled chunk by chunk."""
    index = ShardedKeyIndex(quant, n)
    for lo in range(0, n, 1 << 20):
        index.add(_normal((min(1 << 20, n - lo), d), gen))
    return index


def prepare(case, seed):
    op, d, bits = case["op"], case["d"], case["bits"]
    gen = torch.Generator("cuda").manual_seed(seed)
    state = {"op": op}
    if op in ("append", "prefill", "attend"):
        groups, dtype = case["groups"], _DTYPES[case["dtype"]]
        tokens = {"append": 1, "prefill": case.get("tokens"), "attend": case.get("keys")}[op]
        capacity = 512 if op == "append" else tokens
        state["cache"] = tg.PackedKVCache(_quantizer("prod", d, bits), _quantizer("mse", d, case["vbits"]), groups, capacity)
        keys, values = _cache_rows(groups, tokens, d, gen).to(dtype), _cache_rows(groups, tokens, d, gen).to(dtype)
        if op == "attend":
            state["cache"].append(keys, values)
            state["queries"] = _normal((groups, case["queries"], d), gen).to(dtype)
        else:
            if op == "append":
                keys, values = keys.view(groups, d), values.view(groups, d)
            state["keys"], state["values"] = keys, values
    elif op == "harness":
        host = np.random.default_rng(seed)
        state["mse"], state["prod"] = _quantizer("mse", d, bits), _quantizer("prod", d, bits)
        state["x"] = (host.standard_normal((case["n"], d)) * 3.0).astype(np.float32)
        state["queries"] = (host.standard_normal((case["queries"], d)) * 1.5).astype(np.float32)
    elif op in ("mse", "prod", "sweep"):
        state["quant"] = _quantizer("mse" if op == "mse" else "prod", d, bits)
        state["x"] = _normal((case["n"], d), gen)
        if op == "sweep":
            state["queries"] = _normal((16, d), gen)
    else:
        state["quant"] = _quantizer("prod", d, bits)
        state["index"] = _key_index(state["quant"], case["n"], d, gen)
        state["encoding"] = state["index"].encoding()
        state["queries"] = _normal((d,) if op == "score_one" else (case["queries"], d), gen)
        state["topk"] = case.get("topk")
    return state


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def _packed(encoding):
    return {k: v for k, v in tg.packed_buffers(encoding).items() if v is not None}


def _cache_arrays(cache):
    keys = cache.keys
    return {"codes": keys.codes, "signs": keys.signs, "norms": keys.norms, "residual_norms": keys.residual_norms,
            "value_codes": cache.value_codes, "value_norms": cache.value_norms, "length": keys.length_device}


def run(state):
    op = state["op"]
    if op == "append":
        cache = state["cache"]
        if len(cache) == cache.capacity:      # the sequences are over: the next ones start from an empty cache
            cache.reset()
        cache.append(state["keys"], state["values"])
        return _cache_arrays(cache)
    if op == "prefill":
        state["cache"].reset()
        state["cache"].append(state["keys"], state["values"])
        return _cache_arrays(state["cache"])
    if op == "attend":
        return state["cache"].attend(state["queries"])
    if op == "harness":
        mse, prod, x = state["mse"], state["prod"], state["x"]
        restored = mse.dequantize(mse.quantize(x))
        encoding = prod.quantize(x)
        scores = np.stack([prod.attention_score(q, encoding) for q in state["queries"]])
        return {"restored": restored, "scores": scores}
    quant = state["quant"]
    if op == "mse":
        encoding = quant.quantize(state["x"])
        return dict(_packed(encoding), restored=quant.dequantize(encoding))
    if op == "prod":
        return _packed(quant.quantize(state["x"]))
    if op == "sweep":
        encoding = quant.quantize(state["x"])
        return dict(_packed(encoding), restored=quant.dequantize(encoding),
                    scores=quant.attention_scores(state["queries"], encoding))
    if op == "score_one":
        return quant.attention_score(state["queries"], state["encoding"])
    if op == "scores":
        return quant.attention_scores(state["queries"], state["encoding"])
    top_scores, top_indices = state["index"].search(state["queries"], state["topk"])
    return {"scores": top_scores, "indices": top_indices}


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _mse_bytes(d, bits):
    return d * bits / 8 + 4


def _prod_bytes(d, bits):
    return d * max(bits - 1, 1) / 8 + d / 8 + 8


def work(case):
    op, d, bits = case["op"], case["d"], case["bits"]
    key = _prod_bytes(d, bits)
    if op in ("append", "prefill"):
        # keys: rotation and projection of the residual; values: rotation
        rows = case["groups"] * case.get("tokens", 1)
        element = 4 if case["dtype"] == "float32" else 2
        return {"bytes": rows * (2 * element * d + key + _mse_bytes(d, case["vbits"])), "flops": rows * 6.0 * d * d}
    if op == "attend":
        rows, q = case["groups"] * case["keys"], case["queries"]
        element = 4 if case["dtype"] == "float32" else 2
        return {"bytes": rows * (key + _mse_bytes(d, case["vbits"])) + case["groups"] * q * d * (element + 4.0),
                "flops": rows * q * 6.0 * d}
    n = case["n"]
    if op == "mse":
        return {"bytes": n * (8 * d + 2 * _mse_bytes(d, bits)), "flops": n * 4.0 * d * d}
    if op == "prod":
        return {"bytes": n * (4 * d + key), "flops": n * 4.0 * d * d}
    if op == "sweep":
        return {"bytes": n * (8 * d + 3 * key + 64), "flops": n * (8.0 * d * d + 64 * d)}
    q = case.get("queries", 1)
    if op == "harness":
        return {"bytes": n * (12 * d + 2 * _mse_bytes(d, bits) + (1 + q) * key + 4 * q), "flops": n * (8.0 * d * d + 4 * d * q)}
    if op == "search":
        return {"bytes": n * key + q * case["topk"] * 12.0, "flops": n * 4.0 * d * q}
    return {"bytes": n * (key + 4 * q), "flops": n * 4.0 * d * q}


def tolerance(case):
    if case["op"] in ("append", "prefill", "prod"):
        return {"rel": 1e-6, "max": 1e-5}         # packed bytes are the same; norms are 32-bit sums
    if case["op"] == "search":
        # two keys whose 32-bit scores are equal up to rounding may swap places
        return {"rel": 1e-5, "max": 1e-4, "differ": 2e-3}
    if case["op"] == "attend":
        return {"rel": 2e-5, "max": 2e-4}         # the softmax's exponents carry the scores' 32-bit rounding into the weights
    return {"rel": 1e-5, "max": 1e-4}
