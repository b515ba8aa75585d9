"""CUDA-core decode with a tile per block: more tiles than a cluster has blocks, more blocks than the device holds, pages flushed partially
filled, tokens packed on one side only, every flavour, against attention in 64 bits over the materialized cache."""

import pytest
import torch

import dartkv_b200 as dart

pytestmark = pytest.mark.gpu


def build(batch, heads, dim, chunks, dtype=torch.float32, metadata=torch.float16, seed=0, **cfg):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    base = dict(bits=2, page_size=128, key_group_size=32, value_group_size=32, sink_tokens=2, metadata_dtype=metadata, promote_ratio=0.0)
    base.update(cfg)
    cache = dart.DartKVCache(dart.DartKVCacheConfig(**base))
    for n in chunks:
        cache.append(*(torch.randn(batch, heads, n, dim, generator=gen, device="cuda").to(dtype) for _ in range(2)))
    return cache


def check(cache, rep, flavour=dart.DEQUANT_PER_OP, row_start=None, seed=1):
    batch, heads, tokens, dim = cache.shape
    gen = torch.Generator(device="cuda").manual_seed(seed)
    query = torch.randn(batch, heads * rep, 1, dim, generator=gen, device="cuda")
    out = dart.fused_dart_attention(query, cache, flavour=flavour, row_start=row_start).double().view(batch, heads, rep, dim)
    restored = dart.DEQUANT_PER_OP if flavour == dart.DEQUANT_PER_OP else dart.DEQUANT_FP32      # fp32 caches: nothing is rounded after it
    k, v = (cache._materialize(side, 0, tokens, restored).double() for side in range(2))
    logits = (query.double().view(batch, heads, rep, dim) @ k.transpose(2, 3)) * dim ** -0.5
    if row_start is not None:
        logits = logits.masked_fill(torch.arange(tokens, device="cuda") < row_start.view(batch, 1, 1, 1), float("-inf"))
    ref = torch.softmax(logits, -1) @ v
    assert torch.all((out - ref).abs() <= 1e-5 + 1e-5 * ref.abs()), float((out - ref).abs().max())   # fp32 sums of values up to 5


@pytest.mark.parametrize("tokens", [31, 256, 257, 288, 289, 600, 1024, 1900])
@pytest.mark.parametrize("batch,heads,dim,rep", [(1, 2, 128, 1), (1, 8, 64, 4), (1, 1, 256, 16), (1, 3, 40, 8)])
def test_more_tiles_than_a_cluster(tokens, batch, heads, dim, rep):
    for bits in (2, 8):
        check(build(batch, heads, dim, [tokens], bits=bits, hold_partial_pages=True), rep)


@pytest.mark.parametrize("batch,tokens", [(24, 96), (37, 70), (9, 300), (40, 20)])
def test_more_blocks_than_the_device_holds(batch, tokens):
    cache = build(batch, 8, 64, [tokens])
    check(cache, 4)
    starts = torch.tensor([b * 7 % tokens for b in range(batch)], dtype=torch.int32, device="cuda")
    check(cache, 1, row_start=starts)


@pytest.mark.parametrize("flavour", [dart.DEQUANT_PER_OP, dart.DEQUANT_FP32, dart.DEQUANT_FUSED])
@pytest.mark.parametrize("metadata", [torch.float16, torch.bfloat16, torch.float32])
def test_flavours(flavour, metadata):
    check(build(1, 4, 128, [500], metadata=metadata, bits=4, hold_partial_pages=True), 2, flavour)


@pytest.mark.parametrize("cfg", [dict(), dict(local_tokens=1, value_local_tokens=64), dict(value_local_tokens=200)])
def test_partial_pages_and_tokens_packed_on_one_side(cfg):
    check(build(1, 4, 128, [150] + [1, 40, 7, 130, 90, 1, 1, 33], **cfg), 4)
