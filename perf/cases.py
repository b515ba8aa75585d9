"""Performance cases of the packed KV cache: what a program that serves or evaluates a model asks of it.

Every case goes through the public entry points (``DartKVCache``, ``DartHFCache``, ``fused_dart_attention``,
``streamed_dart_attention``, ``quantize`` / ``quantize_key_mixed`` / ``dequantize``).  Kinds of work:

``decode``    one query token against a resident cache (``fused_dart_attention``)
``verify``    a few query tokens against a resident cache (``streamed_dart_attention``)
``append``    a prompt packed into a new cache, in one chunk or in chunks of ``chunk`` tokens
``update``    a prompt appended to a new cache and the whole cache materialized (``DartKVCache.update``)
``generate``  a prompt and then token after token through the layers of a ``DartHFCache``
``quantize``  keys and values quantized and restored with the functional API

Data as in the benchmark: queries and values are N(0, 1), keys N(0, 1) with one channel in twenty of every KV head
ten times as large.
"""

from __future__ import annotations

import torch

from dartkv_b200 import (DEQUANT_FP32, DEQUANT_FUSED, DEQUANT_PER_OP, DartKVCache, DartKVCacheConfig, dequantize,
                         fused_dart_attention, quantize, quantize_key_mixed, streamed_dart_attention)
from dartkv_b200.integrations import DartHFCache

DTYPE = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}
FLAVOUR = {"per_op": DEQUANT_PER_OP, "fp32": DEQUANT_FP32, "fused": DEQUANT_FUSED}

# The geometry of the long-context workloads: 32 query heads on 8 KV heads of 128 channels, 128-token pages, 2-bit
# values in groups of 64 channels, 2-bit keys in groups of 128 tokens with a quarter of the channels promoted to
# 2+2 bits, 32 dense sink tokens, pages held until they are full.
BASE = dict(query_heads=32, kv_heads=8, head_dim=128, dtype="bf16", metadata="bf16", page=128, sinks=32, hold=True,
            key_bits=2, value_bits=2, key_group=128, value_group=64, promote=0.25)


def _case(kind, name=None, **fields):
    case = dict(BASE, kind=kind, **fields)
    if name is not None:
        case["name"] = name
    return case


def listed():
    return [
        # The smallest call: one query against 256 fp32 tokens, 2-bit in groups of 32, two sinks, partial pages flushed.
        _case("decode", "decode_one_row_fp32", batch=1, tokens=256, query_heads=8, dtype="fp32", metadata="fp16",
              sinks=2, hold=False, key_group=32, value_group=32, promote=0.0, flavour="per_op", padded=False),
        # One layer of an 8B-class model in generation: batch 8, left-padded prompts of unequal length, fp16 scales
        # beside the bf16 cache as the configuration's default has it.
        _case("decode", "decode_layer_left_padded", batch=8, tokens=1163, metadata="fp16", flavour="per_op", padded=True),
        # Decode in a serving batch of ordinary size.
        _case("decode", "decode_batch32_ctx8k", batch=32, tokens=8192, flavour="per_op", padded=False),
        # Long-context decode at the largest batch: 2.9 GB of packed pages per step.
        _case("decode", "decode_batch128_ctx32k", batch=128, tokens=32768, flavour="per_op", padded=False),
        # The 4-bit quality setting in fp16, context not a multiple of the page.
        _case("decode", "decode_4bit_fp16", batch=24, tokens=6001, dtype="fp16", metadata="fp16", key_bits=4,
              value_bits=4, promote=0.0, flavour="per_op", padded=False),
        # The arithmetic of the GPU reference kernels (scale and zero point applied in fp32, nothing rounded).
        _case("decode", "decode_unrounded_ctx16k", batch=16, tokens=16384, flavour="fused", padded=False),
        # Five drafted tokens checked at once against the cache.
        _case("verify", "verify_five_tokens", batch=8, tokens=4096, queries=5),
        # Prefill: a whole prompt packed in one call.
        _case("append", "append_prompt_4k", batch=16, tokens=4096, chunk=4096),
        # The same prompt arriving a page at a time, 4-bit values.
        _case("append", "append_pages_of_128", batch=16, tokens=4096, chunk=128, value_bits=4),
        # A standard attention backend on the packed cache: append, then the dense keys and values back; fp16.
        _case("update", "update_materialize_fp16", batch=4, tokens=2500, dtype="fp16", metadata="fp16"),
        # Prompt and generation through the model-facing cache, fp16 scales beside bf16, across a page boundary.
        _case("generate", "generate_two_layers", batch=8, tokens=1052, metadata="fp16", layers=2, steps=24),
        # The functional quantizer on one layer's keys and values, and back: 1,024 tokens in fp16.
        _case("quantize", "quantize_restore_1k", batch=8, tokens=1024, dtype="fp16", metadata="fp16"),
    ]


def _log(rng, low, high):
    """An integer from low to high, spread over its logarithm."""

    return min(high, max(low, int(round(low * (high / low) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "decode", "verify", "append", "append", "update", "generate", "quantize"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    metadata = rng.choice([dtype, "fp16"])
    kv_heads = rng.choice([2, 4, 8])
    rep = rng.choice([1, 2, 4, 4])
    common = dict(dtype=dtype, metadata=metadata, kv_heads=kv_heads, query_heads=kv_heads * rep,
                  sinks=rng.choice([0, 4, 32, 32]), promote=rng.choice([0.0, 0.125, 0.25, 0.25]),
                  value_group=rng.choice([32, 64, 64, 128]))
    if common["promote"] == 0.0:
        common["key_bits"] = rng.choice([2, 4, 8])
    common["value_bits"] = rng.choice([2, 2, 4, 8])
    if kind == "decode":
        family = rng.choice(["headline", "headline", "headline", "bits", "fp32"])
        if family == "fp32":      # full-precision caches: small heads too, flushed partial pages
            return _case("decode", batch=_log(rng, 1, 4), tokens=_log(rng, 130, 2048), query_heads=8,
                         kv_heads=rng.choice([2, 8]), head_dim=rng.choice([64, 128]), dtype="fp32", metadata="fp16",
                         sinks=rng.choice([2, 32]), hold=rng.choice([True, False]), key_group=rng.choice([32, 128]),
                         value_group=32, promote=0.0, flavour="per_op", padded=False)
        tokens = _log(rng, 200, 32768)
        batch = _log(rng, 1, max(1, min(128, (262144 if family == "bits" else 2 ** 21) // tokens)))
        if family == "headline":
            common.update(key_bits=2, value_bits=2, value_group=rng.choice([64, 64, 128]))
            flavour = rng.choice(["per_op", "per_op", "fused"])
        else:
            flavour = rng.choice(["per_op", "per_op", "fp32"])
        return _case("decode", **common, batch=batch, tokens=tokens, flavour=flavour, padded=rng.random() < 0.25)
    if kind == "verify":
        tokens = _log(rng, 256, 8192)
        return _case("verify", **common, batch=_log(rng, 1, max(1, 32768 // tokens)), tokens=tokens, queries=rng.randint(2, 8))
    if kind == "append":
        tokens = _log(rng, 150, 8192)
        return _case("append", **common, batch=_log(rng, 1, max(1, 65536 // tokens)), tokens=tokens,
                     chunk=rng.choice([tokens, tokens, 128, 512]) if tokens > 512 else tokens)
    if kind == "update":
        tokens = _log(rng, 150, 4096)
        return _case("update", **common, batch=_log(rng, 1, max(1, 10000 // tokens)), tokens=tokens,
                     hold=rng.choice([True, True, False]))
    if kind == "generate":
        tokens = _log(rng, 100, 2048)
        return _case("generate", **common, batch=_log(rng, 1, max(1, 16384 // tokens)), tokens=tokens, layers=rng.randint(1, 2),
                     steps=rng.randint(4, 24))
    tokens = _log(rng, 100, 4096)
    return _case("quantize", **common, batch=_log(rng, 1, max(1, 8192 // tokens)), tokens=tokens,
                 key_group=rng.choice([32, 64, 128]))


# ------------------------------------------------------------------------------------------------ inputs
def _config(case):
    return DartKVCacheConfig(bits=case["value_bits"], key_bits=case["key_bits"], value_bits=case["value_bits"],
                             key_group_size=case["key_group"], value_group_size=case["value_group"],
                             page_size=case["page"], sink_tokens=case["sinks"], hold_partial_pages=case["hold"],
                             promote_ratio=case["promote"], metadata_dtype=DTYPE[case["metadata"]])


class _Data:
    def __init__(self, case, seed):
        self.case = case
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        heads, channels = case["kv_heads"], case["head_dim"]
        self.factor = torch.ones(heads, 1, channels, dtype=DTYPE[case["dtype"]], device="cuda")
        scores = torch.rand(heads, channels, generator=self.gen, device="cuda")
        outliers = scores.topk(channels // 20, dim=-1).indices
        self.factor.view(heads, channels).scatter_(1, outliers, 10.0)

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.gen, dtype=DTYPE[self.case["dtype"]], device="cuda")

    def keys(self, tokens):
        c = self.case
        return self.normal(c["batch"], c["kv_heads"], tokens, c["head_dim"]) * self.factor

    def values(self, tokens):
        c = self.case
        return self.normal(c["batch"], c["kv_heads"], tokens, c["head_dim"])

    def projected(self, tokens):
        """Keys and values as a model's projections leave them: ``[B, T, H, D]`` seen as ``[B, H, T, D]``."""

        return [x.transpose(1, 2).contiguous().transpose(1, 2) for x in (self.keys(tokens), self.values(tokens))]

    def query(self, tokens=1):
        c = self.case
        return self.normal(c["batch"], c["query_heads"], tokens, c["head_dim"])


def prepare(case, seed):
    data = _Data(case, seed)
    state = {"case": case, "kind": case["kind"], "config": _config(case), "tokens": case["tokens"]}
    if case["kind"] in ("decode", "verify"):
        # the resident cache: the prompt came in earlier
        cache = DartKVCache(state["config"], max_tokens=case["tokens"] + 256)
        done = 0
        while done < case["tokens"]:
            step = min(case["tokens"] - done, case["sinks"] + 1024 if done == 0 else 1024)
            cache.append(data.keys(step), data.values(step))
            done += step
        state["cache"] = cache
        state["query"] = data.query(case.get("queries", 1))
        state["scale"] = case["head_dim"] ** -0.5
        if case["kind"] == "decode":
            state["flavour"] = FLAVOUR[case["flavour"]]
            if case["padded"]:
                pads = torch.rand(case["batch"], generator=data.gen, device="cuda") * (case["tokens"] // 2)
                pads[0] = 0
                state["row_start"] = pads.to(torch.int32)
    elif case["kind"] in ("append", "update"):
        state["keys"], state["values"] = data.keys(case["tokens"]), data.values(case["tokens"])
    elif case["kind"] == "generate":
        layers = range(case["layers"])
        state["prompts"] = [data.projected(case["tokens"]) for _ in layers]
        state["steps"] = [[(data.query(), *data.projected(1)) for _ in layers] for _ in range(case["steps"])]
        state["scale"] = case["head_dim"] ** -0.5
    else:
        state["keys"], state["values"] = data.keys(case["tokens"]), data.values(case["tokens"])
    return state


# ------------------------------------------------------------------------------------------------ one pass
def _contents(cache):
    """The packed pages, packed value rows and dense tokens of a cache, as views of what has been written."""

    config, pools, seen = cache.config, cache._pools, cache.seen_tokens
    sinks = min(seen, config.sink_tokens)
    pages = (seen - sinks) // config.page_size
    rows = pages * config.page_size
    ring = pools["k_ring"].shape[2]
    first, end = (sinks + rows) % ring, seen % ring
    pending = seen - sinks - rows
    parts = [(first, first + pending)] if first + pending <= ring else [(first, ring), (0, end)]
    out = [pools["k_pages"][:, :, :pages], pools["v_codes"][:, :, :rows], pools["v_meta"][:, :, :rows]]
    for name in ("k_sink", "v_sink"):
        out.append(pools[name][:, :, :sinks])
    for name in ("k_ring", "v_ring"):
        out.extend(pools[name][:, :, a:b] for a, b in parts)
    return out


def run(state):
    kind = state["kind"]
    if kind == "decode":
        return fused_dart_attention(state["query"], state["cache"], scale=state["scale"], flavour=state["flavour"],
                                    row_start=state.get("row_start"))
    if kind == "verify":
        return streamed_dart_attention(state["query"], state["cache"], scale=state["scale"])
    if kind == "append":
        cache = DartKVCache(state["config"], max_tokens=state["tokens"])
        keys, values, chunk = state["keys"], state["values"], state["case"]["chunk"]
        if chunk >= state["tokens"]:
            cache.append(keys, values)
        else:
            for start in range(0, state["tokens"], chunk):
                cache.append(keys[:, :, start:start + chunk], values[:, :, start:start + chunk])
        return _contents(cache)
    if kind == "update":
        return DartKVCache(state["config"]).update(state["keys"], state["values"])
    if kind == "generate":
        cache = DartHFCache(state["config"], max_tokens=state["tokens"] + len(state["steps"]))
        fused = {"dart_fused_attention": True}
        for layer, (keys, values) in enumerate(state["prompts"]):
            cache.update(keys, values, layer, fused)
        out = []
        for step in state["steps"]:
            for layer, (query, keys, values) in enumerate(step):
                out.append(cache.decode_step(query, keys, values, layer, scale=state["scale"]))
        return out + _contents(cache.layer_for_attention(0))
    case, md = state["case"], DTYPE[state["case"]["metadata"]]
    if case["promote"] > 0.0:
        keys = quantize_key_mixed(state["keys"], group_size=case["key_group"], promote_ratio=case["promote"], metadata_dtype=md)
        key_fields = [keys.low_values, keys.high_values, keys.channel_indices, keys.scale, keys.zero_point]
    else:
        keys = quantize(state["keys"], bits=case["key_bits"], group_size=case["key_group"], metadata_dtype=md, axis=-2)
        key_fields = [keys.values, keys.scale, keys.zero_point]
    values = quantize(state["values"], bits=case["value_bits"], group_size=case["value_group"], metadata_dtype=md)
    restored_keys = keys.dequantize()
    return key_fields + [values.values, values.scale, values.zero_point, restored_keys, dequantize(values)]


# ------------------------------------------------------------------------------------------------ necessary work
def _token_bytes(case):
    """Packed bytes of one token of one KV head (key and value codes, scales and zero points), and its dense bytes."""

    d, md = case["head_dim"], BYTES[case["metadata"]]
    groups = -(-d // case["value_group"])
    value = d * case["value_bits"] / 8 + 2 * groups * md
    if case["promote"] > 0.0:
        promoted = int(d * case["promote"] + 1e-6)
        key = (d + promoted) * 2 / 8 + (4 * promoted) / case["page"] + 2 * d * md / case["key_group"]
    else:
        key = d * case["key_bits"] / 8 + 2 * d * md / case["key_group"]
    return key + value, 2 * d * BYTES[case["dtype"]]


def _cache_bytes(case, tokens):
    """Bytes of a cache of that many tokens: dense sinks, packed pages, dense tail where partial pages are held."""

    packed, dense = _token_bytes(case)
    sinks = min(tokens, case["sinks"])
    tail = (tokens - sinks) % case["page"] if case["hold"] else 0
    return case["batch"] * case["kv_heads"] * ((tokens - sinks - tail) * packed + (sinks + tail) * dense)


def work(case):
    rows = case["batch"] * case["kv_heads"]
    tokens, d = case["tokens"], case["head_dim"]
    dense = rows * tokens * _token_bytes(case)[1]
    attention = 4.0 * case["batch"] * case["query_heads"] * d      # flops per query token and cached token
    vectors = 2 * case["batch"] * case["query_heads"] * d * BYTES[case["dtype"]]
    kind = case["kind"]
    if kind in ("decode", "verify"):
        queries = case.get("queries", 1)
        live = 0.75 if case.get("padded") else 1.0                 # left padding: a quarter of the tokens on average
        return {"bytes": live * _cache_bytes(case, tokens) + queries * vectors, "flops": live * queries * attention * tokens}
    quantizing = 8.0 * rows * tokens * 2 * d                       # min, max, subtract, divide, round, clamp, pack
    if kind == "append":
        return {"bytes": dense + _cache_bytes(case, tokens), "flops": quantizing}
    if kind == "update":
        return {"bytes": 2 * dense + _cache_bytes(case, tokens), "flops": quantizing + 2.0 * rows * tokens * 2 * d}
    if kind == "generate":
        prompt = dense + _cache_bytes(case, tokens)
        steps = sum(_cache_bytes(case, tokens + i + 1) + vectors + 2 * rows * _token_bytes(case)[1] for i in range(case["steps"]))
        flops = quantizing + sum(attention * (tokens + i + 1) for i in range(case["steps"]))
        return {"bytes": case["layers"] * (prompt + steps), "flops": case["layers"] * flops}
    return {"bytes": 2 * dense + 2 * rows * tokens * _token_bytes(case)[0], "flops": quantizing + 2.0 * rows * tokens * 2 * d}


def tolerance(case):
    if case["kind"] in ("append", "update", "quantize"):
        return "exact"           # packed codes, scales, zero points and restored values
    if case["dtype"] == "fp32":
        return {"rel": 1e-5, "max": 1e-4}
    if case.get("flavour") == "fused":
        # the weights q*scale and p*scale travel as 16-bit numbers
        return {"rel": 1e-2, "max": 5e-2}
    # fp32 sums, one rounding of the result to the 16-bit type: at most an ulp apart where two results straddle a tie
    return {"rel": 4e-3, "max": 2e-2} if case["dtype"] == "bf16" else {"rel": 1e-3, "max": 5e-3}
