"""The CUDA-core decode kernel for few tokens in uniform key pages (a block per 32 tokens, the blocks of a KV head one cluster of
up to eight) and its border to the kernel of longer caches at 256 tokens, against attention in 64 bits over the materialized cache."""

import pytest
import torch

import dartkv_b200 as dart

pytestmark = pytest.mark.gpu

# bits, metadata dtype and cache dtype go with the channels, so that every variant of each is met
SHAPES = [(24, 2, torch.float16, torch.float32), (40, 4, torch.bfloat16, torch.float32), (96, 8, torch.float32, torch.float32),
          (128, 2, torch.float16, torch.bfloat16), (200, 2, torch.float32, torch.float16), (256, 4, torch.float16, torch.float32)]


def make(keys, values, step, **config):
    cache = dart.DartKVCache(dart.DartKVCacheConfig(**dict(dict(bits=2, page_size=128, key_group_size=32, value_group_size=8, sink_tokens=2),
                                                           **config)))
    for start in range(0, keys.shape[2], step):
        cache.append(keys[:, :, start:start + step], values[:, :, start:start + step])
    return cache


def reference(query, cache, start=None):
    k, v = (t.double() for t in cache.get())
    rep = query.shape[1] // k.shape[1]
    logits = query.double().view(k.shape[0], k.shape[1], rep, -1) @ k.transpose(2, 3) * k.shape[-1] ** -0.5
    if start is not None:
        logits = logits.masked_fill(torch.arange(k.shape[2], device="cuda") < start.view(-1, 1, 1, 1), float("-inf"))
    return (torch.softmax(logits, -1) @ v).view(query.shape)


@pytest.mark.parametrize("head_dim,bits,metadata,dtype", SHAPES)
@pytest.mark.parametrize("tokens", [1, 2, 31, 33, 64, 130, 161, 225, 256, 257])
@pytest.mark.parametrize("hold", [True, False])
def test_few_tokens(head_dim, bits, metadata, dtype, tokens, hold):
    gen = torch.Generator(device="cuda").manual_seed(head_dim + tokens)
    keys, values = (torch.randn(2, 2, tokens, head_dim, generator=gen, device="cuda").to(dtype) for _ in range(2))
    cache = make(keys, values, 100, bits=bits, metadata_dtype=metadata, hold_partial_pages=hold)
    starts = [None, torch.tensor([tokens // 3, tokens - 1], dtype=torch.int32, device="cuda"),
              torch.tensor([0, min(tokens - 1, 70)], dtype=torch.int32, device="cuda")]   # whole tiles before the first live token
    for rep in (1, 3, 5, 16):
        query = torch.randn(2, 2 * rep, 1, head_dim, generator=gen, device="cuda")
        for start in starts:
            out = dart.fused_dart_attention(query, cache, row_start=start)
            # fp32 sums over at most 257 weights that add up to one, of values up to 5: 1e-5 as for the other fp32 checks
            assert (out.double() - reference(query, cache, start)).abs().max() < 1e-5


@pytest.mark.parametrize("step", [9, 8, 5, 3])   # pages of that many tokens: fewer than, as many as and more than a warp has lanes
def test_many_irregular_pages(step):
    gen = torch.Generator(device="cuda").manual_seed(step)
    keys, values = (torch.randn(1, 2, 2 + 254, 128, generator=gen, device="cuda") for _ in range(2))
    cache = make(keys, values, step, sink_tokens=0)
    for flavour in (dart.DEQUANT_PER_OP, dart.DEQUANT_FP32):
        for rep in (1, 4):
            query = torch.randn(1, 2 * rep, 1, 128, generator=gen, device="cuda")
            # fp16 scales: the two flavours restore fp32 data differently; get() is the per-op one, whose roundings are 2^-11
            bound = 1e-5 if flavour == dart.DEQUANT_PER_OP else 2e-2
            assert (dart.fused_dart_attention(query, cache, flavour=flavour).double() - reference(query, cache)).abs().max() < bound


@pytest.mark.parametrize("hold", [True, False])
@pytest.mark.parametrize("tokens", [[0, 1], [0, 2], [2, 34], [5, 6], [40, 41], [64, 96], [200, 256], [255, 256], [0, 256]])
def test_nan_keys(tokens, hold):
    # dense: NaN.  Packed: one Inf in every group of 32 keys, which makes the group's scale infinite and all of them NaN (0 * Inf; a
    # group of Inf only has no range and restores to Inf); wherever the tiles are cut
    gen = torch.Generator(device="cuda").manual_seed(7)
    keys, values = (torch.randn(2, 2, 256, 128, generator=gen, device="cuda") for _ in range(2))
    dense = range(tokens[0], tokens[1] if hold else min(tokens[1], 2))
    keys[1, 1, list(dense), 9] = float("nan")
    keys[1, 1, list(range(max(tokens[0], dense.stop), tokens[1], 32)), 9] = float("inf")
    cache = make(keys, values, 256, hold_partial_pages=hold, page_size=512 if hold else 128)
    query = torch.randn(2, 8, 1, 128, generator=gen, device="cuda")
    out = dart.fused_dart_attention(query, cache)
    assert out[1, 4:].isnan().all()
    ref = reference(query, cache)
    out[1, 4:] = ref[1, 4:] = 0.0
    assert (out.double() - ref).abs().max() < 1e-5


@pytest.mark.parametrize("tokens", [[0, 32], [32, 64], [3, 4], [64, 256], [224, 256]])
def test_infinitely_small_logits_weigh_nothing(tokens):
    gen = torch.Generator(device="cuda").manual_seed(8)
    keys, values = (torch.randn(1, 2, 256, 128, generator=gen, device="cuda") for _ in range(2))
    query = torch.rand(1, 8, 1, 128, generator=gen, device="cuda") + 0.5
    keys[:, 1, tokens[0]:tokens[1], 9] = float("-inf")
    cache = make(keys, values, 256, hold_partial_pages=True, page_size=512)
    assert (dart.fused_dart_attention(query, cache).double() - reference(query, cache)).abs().max() < 1e-5


@pytest.mark.parametrize("token", [0, 31, 100, 255])
def test_a_value_whose_weight_underflows_still_counts(token):
    keys, values = torch.ones(1, 2, 256, 128, device="cuda"), torch.ones(1, 2, 256, 128, device="cuda")
    keys[:, :, token] = 0
    values[:, 1, token, 5] = float("nan")
    out = dart.fused_dart_attention(torch.full((1, 8, 1, 128), 12.0, device="cuda"), make(keys, values, 256, hold_partial_pages=True, page_size=512))
    assert out[:, 4:, :, 5].isnan().all()
    out[:, 4:, :, 5] = 1.0
    assert torch.allclose(out, torch.ones_like(out), atol=1e-5)
