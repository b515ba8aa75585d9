"""Nine to 64 query rows per KV head in calls large enough for the blocks that restore a page once for all rows, at the edges of the row groups, of the chunks
of dense tokens and of the blocks' shares, against attention in 64 bits over the materialized cache."""

import ctypes

import pytest
import torch

import dartkv_b200 as dart
from dartkv_b200 import _lib

pytestmark = pytest.mark.gpu


def assert_restored_once_for_all_rows(cache, dtype, rows):
    info, (_, heads, tokens, _) = _lib.DecodePlanInfo(), cache.shape
    _lib.check(_lib.LIB.dartkv_decode_plan_rows(ctypes.byref(cache.descriptor), _lib.DTYPE_CODE[dtype], heads * rows, _lib.DEQUANT_PER_OP, tokens,
                                                ctypes.byref(info)))
    assert info.kernel == 4 and info.unit_pages == 0


def check(cache, dtype, rows, seed, row_start=None, once=True):
    if once:
        assert_restored_once_for_all_rows(cache, dtype, rows)
    batch, heads, tokens, _ = cache.shape
    gen = torch.Generator(device="cuda").manual_seed(seed)
    query = torch.randn(batch, heads * rows, 1, 128, generator=gen, device="cuda", dtype=dtype)
    out = dart.fused_dart_attention(query, cache, fallback=False, row_start=row_start).double().view(batch, heads, rows, 128)
    assert cache.decode_status() == 0
    k, v = (t.double() for t in cache.get())
    logits = (query.double().view(batch, heads, rows, 128) @ k.transpose(2, 3)) * 128 ** -0.5
    if row_start is not None:
        logits = logits.masked_fill(torch.arange(tokens, device="cuda") < row_start.view(batch, 1, 1, 1), float("-inf"))
    ref = torch.softmax(logits, -1) @ v
    half_ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11      # of a result: at most this share of it
    assert torch.all((out - ref).abs() <= ref.abs() * half_ulp + 4e-5), float((out - ref).abs().max())   # fp32 sums of values up to 5


def build(dtype, metadata, tokens, batch=2, sinks=32, seed=0, chunks=None, **cfg):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    base = dict(bits=2, page_size=128, key_group_size=128, value_group_size=64, sink_tokens=sinks, hold_partial_pages=True)
    base.update(cfg)
    cache = dart.DartKVCache(dart.DartKVCacheConfig(metadata_dtype=metadata, **base))
    for n in chunks or [tokens]:
        keys, values = (torch.randn(batch, 2, n, 128, generator=gen, device="cuda", dtype=dtype) for _ in range(2))
        cache.append(keys, values)
    return cache


@pytest.mark.parametrize("key_bits,value_bits,promote,value_group", [(2, 2, 0.25, 64), (2, 4, 0.0, 32), (2, 8, 0.1, 128), (4, 2, 0.0, 64),
                                                                   (4, 4, 0.0, 16), (4, 8, 0.0, 128), (2, 2, 1.0, 64)])
@pytest.mark.parametrize("dtype,metadata", [(torch.bfloat16, torch.bfloat16), (torch.float16, torch.float16), (torch.bfloat16, torch.float16)])
def test_rows_and_code_widths(dtype, metadata, key_bits, value_bits, promote, value_group):
    cache = build(dtype, metadata, 32 + 9 * 128 + 45, batch=37, key_bits=key_bits, value_bits=value_bits, promote_ratio=promote, value_group_size=value_group)
    for rows in (9, 16, 17, 24, 25, 32, 33, 64):
        check(cache, dtype, rows, rows, once=(key_bits, value_bits) != (4, 8))   # those pages go through in passes of four rows


@pytest.mark.parametrize("sinks,tail", [(0, 0), (0, 1), (0, 127), (32, 95), (32, 96), (32, 97), (4, 127), (200, 0), (300, 127)])
def test_dense_tokens(sinks, tail):
    cache = build(torch.bfloat16, torch.bfloat16, sinks + 8 * 128 + tail, batch=40, sinks=sinks, promote_ratio=0.25)
    check(cache, torch.bfloat16, 20, sinks + tail)


@pytest.mark.parametrize("batch,pages", [(16, 61), (16, 17), (40, 9), (75, 8)])
def test_shares_of_the_blocks_and_left_padding(batch, pages):
    tokens = 32 + 128 * pages + 70
    cache = build(torch.float16, torch.float16, tokens, batch=batch, bits=4)
    check(cache, torch.float16, 12, pages)
    starts = torch.tensor([(b * 977 + 31) % (tokens - 1) for b in range(batch - 1)] + [tokens - 1], dtype=torch.int32, device="cuda")
    check(cache, torch.float16, 12, pages, starts)


@pytest.mark.parametrize("promote,window", [(0.25, 128), (0.0, 64), (0.1, 300)])
def test_tokens_packed_on_one_side_only(promote, window):
    cache = build(torch.bfloat16, torch.float16, 0, batch=40, promote_ratio=promote, local_tokens=1, value_local_tokens=window,
                  chunks=[32 + 8 * 128 + 40] + [1] * 30)
    check(cache, torch.bfloat16, 18, window)


@pytest.mark.parametrize("promote,metadata", [(0.25, torch.bfloat16), (0.1, torch.float16)])
def test_left_padding_with_promoted_channels(promote, metadata):
    # blocks that begin behind a row's first pages, whose promoted channels differ from page to page
    tokens, batch = 32 + 128 * 9 + 70, 40
    cache = build(torch.bfloat16, metadata, tokens, batch=batch, promote_ratio=promote)
    starts = torch.tensor([(b * 977 + 31) % (tokens - 1) for b in range(batch - 1)] + [tokens - 1], dtype=torch.int32, device="cuda")
    for rows in (12, 20, 30):
        check(cache, torch.bfloat16, rows, rows, starts)


def make(dtype, keys, values, **cfg):
    base = dict(bits=2, page_size=128, key_group_size=128, value_group_size=64, sink_tokens=32, hold_partial_pages=True, metadata_dtype=dtype)
    base.update(cfg)
    cache = dart.DartKVCache(dart.DartKVCacheConfig(**base))
    cache.append(keys, values)
    return cache


def data(dtype, tokens, seed, batch=40):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(batch, 2, tokens, 128, generator=gen, device="cuda", dtype=dtype) for _ in range(2)]


@pytest.mark.parametrize("dtype,cfg", [(torch.bfloat16, dict(promote_ratio=0.25)), (torch.float16, dict(bits=4))])
@pytest.mark.parametrize("rows", [9, 20, 32])
@pytest.mark.parametrize("first,last,bad", [(32 + 5, 33 + 5, "inf"), (32 + 128 * 4, 33 + 128 * 4, "inf"), (31 + 128 * 9, 32 + 128 * 9, "inf"),   # a page of NaN logits
                                            (0, 32, "nan"), (3, 4, "nan"), (-45, -20, "nan"), (-1, None, "nan")])                                 # dense tokens
def test_nan_logits_reach_the_output(dtype, cfg, rows, first, last, bad):
    # an Inf makes the scale of its channel infinite: every key of the page has a NaN (0 * Inf) there
    keys, values = data(dtype, 32 + 9 * 128 + 45, rows)
    keys[7, 1, first:last, 9] = float(bad)
    cache = make(dtype, keys, values, **cfg)
    assert_restored_once_for_all_rows(cache, dtype, rows)
    query = torch.randn(40, 2 * rows, 1, 128, device="cuda", dtype=dtype)
    out = dart.fused_dart_attention(query, cache, fallback=False).view(40, 2, rows, 128)
    assert out[7, 1].isnan().all()
    out[7, 1] = 0
    assert out.isfinite().all() and cache.decode_status() == 0


@pytest.mark.parametrize("bad", ["nan", "inf"])
@pytest.mark.parametrize("rows", [9, 24, 32])
def test_a_value_whose_weight_underflows_still_counts(rows, bad):
    # the sink tokens' logits are 0, the others' 12 * sqrt(128): their weight is zero in fp32, and zero * bad is NaN
    keys, values = (torch.ones(40, 2, 32 + 9 * 128, 128, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    keys[:, :, :32] = 0
    values[7, 1, 7, 5] = float(bad)
    cache = make(torch.bfloat16, keys, values, promote_ratio=0.25)
    assert_restored_once_for_all_rows(cache, torch.bfloat16, rows)
    query = torch.full((40, 2 * rows, 1, 128), 12.0, device="cuda", dtype=torch.bfloat16)
    out = dart.fused_dart_attention(query, cache, fallback=False).float().view(40, 2, rows, 128)
    assert out[7, 1, :, 5].isnan().all()
    out[7, 1, :, 5] = 1.0
    assert torch.allclose(out, torch.ones_like(out), atol=1e-2)


@pytest.mark.parametrize("dtype,cfg", [(torch.bfloat16, dict(promote_ratio=0.25)), (torch.float16, dict(bits=4))])
@pytest.mark.parametrize("rows", [9, 20, 32])
def test_infinitely_small_logits_of_dense_tokens_weigh_nothing(dtype, cfg, rows):
    keys, values = data(dtype, 32 + 9 * 128 + 3, rows)
    query = torch.rand(40, 2, rows, 128, device="cuda") + 0.5
    keys[:, :, :32, 4] = float("-inf")
    keys[:, :, -1, 4] = float("-inf")
    cache = make(dtype, keys, values, **cfg)
    assert_restored_once_for_all_rows(cache, dtype, rows)
    query = query.to(dtype)
    out = dart.fused_dart_attention(query.view(40, 2 * rows, 1, 128), cache, fallback=False).double().view(40, 2, rows, 128)
    k, v = (t.double() for t in cache.get())
    ref = torch.softmax(query.double() @ k.transpose(2, 3) * 128 ** -0.5, -1) @ v
    half_ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert torch.all((out - ref).abs() <= ref.abs() * half_ulp + 4e-5), float((out - ref).abs().max())   # as in check()
