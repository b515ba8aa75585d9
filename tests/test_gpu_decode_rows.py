"""More than four query rows per KV head in one launch (several query tokens at once, wide query groups) against the
oracle's streamed attention on seeded inputs."""

import numpy as np
import pytest
import torch

import dartkv_b200 as dart
from dartkv_b200 import _lib
from dartkv_b200.synthetic import make_kvq
from oracle import dartkv_oracle as orc
from tests.helpers import DT_TAG, to_np

pytestmark = pytest.mark.gpu


def build(dtype, metadata, batch, heads, tokens, chunks=None, seed=0, **cfg):
    tag = DT_TAG[dtype]
    keys, values, _ = make_kvq(seed, batch, heads, tokens, 128, query_heads=heads, dtype=dtype, outlier_fraction=0.05)
    base = dict(bits=2, page_size=128, key_group_size=128, value_group_size=64, sink_tokens=32, hold_partial_pages=True)
    base.update(cfg)
    cache = dart.DartKVCache(dart.DartKVCacheConfig(metadata_dtype=metadata, **base))
    oracle = orc.OracleCache(orc.CacheConfig(metadata_dtype=DT_TAG[metadata], **base), tag)
    start = 0
    for chunk in chunks or [tokens]:
        cache.append(keys[:, :, start:start + chunk].cuda(), values[:, :, start:start + chunk].cuda())
        oracle.append(to_np(keys[:, :, start:start + chunk]), to_np(values[:, :, start:start + chunk]))
        start += chunk
    return cache, oracle


def check(cache, oracle, dtype, hq, queries, seed=0, row_start=None, call=None):
    tag = DT_TAG[dtype]
    batch = cache.shape[0]
    query = torch.randn(batch, hq, queries, 128, generator=torch.Generator().manual_seed(seed + 1000)).to(dtype)
    out = call(query.cuda()) if call else dart.streamed_dart_attention(query.cuda(), cache)
    assert cache.decode_status() == 0
    ref32 = orc.streamed_attention(to_np(query), oracle, tag, return_f32=True,
                                   row_start=None if row_start is None else np.asarray(row_start))
    got = to_np(out)
    assert got.shape == ref32.shape
    # one rounding of an fp32 result to the 16-bit output: half an ulp, and the fp32 sums' own order
    ulp = np.abs(ref32) * (2.0 ** -8 if tag == "bf16" else 2.0 ** -11)
    assert np.all(np.abs(got - ref32) <= ulp + 2e-5), float(np.abs(got - ref32).max())


GEOMETRIES = [dict(promote_ratio=0.25), dict(promote_ratio=0.1, value_group_size=16), dict(), dict(bits=4),
              dict(bits=4, promote_ratio=1.0, value_group_size=128), dict(key_bits=4, value_bits=2, value_group_size=32),
              dict(bits=8, promote_ratio=0.25), dict(key_bits=2, value_bits=8, value_group_size=32)]


@pytest.mark.parametrize("dtype,metadata", [(torch.bfloat16, torch.bfloat16), (torch.float16, torch.float16),
                                            (torch.bfloat16, torch.float16), (torch.float16, torch.bfloat16)])
@pytest.mark.parametrize("cfg", GEOMETRIES)
def test_query_tokens_share_a_launch(dtype, metadata, cfg):
    cache, oracle = build(dtype, metadata, 2, 2, 32 + 8 * 128 + 77, seed=3, **cfg)
    assert cache.decode_rows_limit(dtype, _lib.DEQUANT_PER_OP, cache.seen_tokens) == 64
    check(cache, oracle, dtype, 8, 5)      # 4 heads x 5 tokens: three groups of 7, 7 and 6 rows
    check(cache, oracle, dtype, 8, 17)     # 68 rows: two calls
    check(cache, oracle, dtype, 8, 2)      # 8 rows: two passes
    check(cache, oracle, dtype, 2, 9)      # one head per KV head: groups of 5 and 4 rows
    check(cache, oracle, dtype, 6, 6)      # 18 rows: three groups of six


@pytest.mark.parametrize("rep", [5, 8, 9, 16, 20])
def test_wide_query_groups(rep):
    cache, oracle = build(torch.bfloat16, torch.bfloat16, 2, 2, 32 + 9 * 128 + 3, seed=4, promote_ratio=0.25)
    for _ in range(2):                     # through Python first, through the native host path after
        check(cache, oracle, torch.bfloat16, 2 * rep, 1, call=lambda q: dart.fused_dart_attention(q, cache, fallback=False))


@pytest.mark.parametrize("tokens", [1023, 1024, 32 + 8 * 128, 32 + 8 * 128 + 1, 32 + 17 * 128 + 127])
def test_edges_of_sinks_pages_and_units(tokens):
    cache, oracle = build(torch.float16, torch.float16, 1, 2, tokens, seed=5, bits=4)
    check(cache, oracle, torch.float16, 8, 3)


@pytest.mark.parametrize("split", ["aligned", "unaligned:5"])
def test_both_split_families_and_left_padding(split, decode_split):
    decode_split(split)
    starts = [0, 33, 32 + 128 + 7, 32 + 5 * 128 + 121, 32 + 11 * 128 + 8]
    cache, oracle = build(torch.bfloat16, torch.float16, len(starts), 2, 32 + 11 * 128 + 9, seed=6, promote_ratio=0.25)
    rows = torch.tensor(starts, dtype=torch.int32).cuda()
    check(cache, oracle, torch.bfloat16, 24, 1, row_start=starts,
          call=lambda q: dart.fused_dart_attention(q, cache, fallback=False, row_start=rows))


def test_tokens_packed_on_one_side_only():
    cache, oracle = build(torch.float16, torch.float16, 1, 2, 32 + 8 * 128 + 40 + 30, seed=7, bits=4, local_tokens=1,
                          value_local_tokens=128, chunks=[32 + 8 * 128 + 40] + [1] * 30)
    check(cache, oracle, torch.float16, 8, 4)


def test_scratch_of_calls_of_many_widths_is_shared():
    cache, oracle = build(torch.bfloat16, torch.bfloat16, 2, 2, 32 + 8 * 128 + 5, seed=8, promote_ratio=0.25)
    for queries in (1, 3, 5, 9, 2, 12, 16, 1, 16):
        check(cache, oracle, torch.bfloat16, 8, queries)
    largest = cache.decode_workspace(2 * 64)[0].numel()
    assert sum(buffer.numel() for buffer in cache._scratch) <= 2 * largest
