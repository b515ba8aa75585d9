"""Inf and NaN in a cache reach the attention output as in softmax(q k) v, whichever split of the work they fall into."""

import pytest
import torch

import dartkv_b200 as dart

pytestmark = pytest.mark.gpu

CONFIGS = [(torch.float32, dict(bits=2, key_group_size=32, value_group_size=32, promote_ratio=0.0)),
           (torch.bfloat16, dict(bits=2, key_group_size=128, value_group_size=64, promote_ratio=0.25)),
           (torch.float16, dict(bits=4, key_group_size=128, value_group_size=64, promote_ratio=0.0))]


def make(dtype, cfg, keys, values):
    cache = dart.DartKVCache(dart.DartKVCacheConfig(page_size=128, sink_tokens=32, hold_partial_pages=True, metadata_dtype=torch.float16,
                                                    **cfg))
    cache.append(keys.to(dtype).cuda(), values.to(dtype).cuda())
    return cache


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("dtype,cfg", CONFIGS)
def test_a_value_whose_weight_underflows_still_counts(dtype, cfg, bad):
    # the sink tokens' logits are 0, the others' 12 * sqrt(128): their weight is zero in fp32, and zero * bad is NaN.
    # No token follows the full pages, so the sinks are a split of their own under every kernel
    keys, values = torch.ones(1, 2, 32 + 3 * 128, 128), torch.ones(1, 2, 32 + 3 * 128, 128)
    keys[:, :, :32] = 0
    values[:, 1, 7, 5] = bad
    cache = make(dtype, cfg, keys, values)
    query = torch.full((1, 8, 1, 128), 12.0, device="cuda", dtype=dtype)
    for _ in range(2):
        out = dart.fused_dart_attention(query, cache).float()
        assert out[:, 4:, :, 5].isnan().all()
        out[:, 4:, :, 5] = 1.0
        assert torch.allclose(out, torch.ones_like(out), atol=1e-2)


@pytest.mark.parametrize("tokens", [[0, 32], [3, 4], [32 + 4 * 128, 32 + 4 * 128 + 3], [32 + 4 * 128 + 2, 32 + 4 * 128 + 3]])
def test_nan_keys_of_the_cuda_core_kernel(tokens):
    # dense tokens, wherever the splits are cut: runs of NaN logits only, and single ones
    gen = torch.Generator().manual_seed(2)
    keys, values = torch.randn(1, 2, 32 + 4 * 128 + 3, 128, generator=gen), torch.randn(1, 2, 32 + 4 * 128 + 3, 128, generator=gen)
    keys[:, 1, tokens[0]:tokens[1], 9] = float("nan")
    cache = make(*CONFIGS[0], keys, values)
    query = torch.randn(1, 8, 1, 128, generator=gen).cuda()
    out = dart.fused_dart_attention(query, cache)
    assert out[:, 4:].isnan().all() and out[:, :4].isfinite().all()


def test_infinitely_small_logits_weigh_nothing():
    gen = torch.Generator().manual_seed(3)
    keys, values = torch.randn(1, 1, 32 + 2 * 128 + 3, 128, generator=gen), torch.randn(1, 1, 32 + 2 * 128 + 3, 128, generator=gen)
    query = torch.rand(1, 2, 1, 128, generator=gen).cuda() + 0.5
    keys[:, :, :32, 4] = float("-inf")      # a whole split
    keys[:, :, -1, 4] = float("-inf")       # one token of another
    cache = make(*CONFIGS[0], keys, values)
    k, v = cache.get()
    ref = torch.softmax(query.double() @ k.double().transpose(2, 3) * 128 ** -0.5, -1) @ v.double()
    assert (dart.fused_dart_attention(query, cache).double() - ref).abs().max() < 1e-5


# the two kernels of 2-bit pages, the kernel of 4-bit pages (decode_rows.cu) and that of 8-bit keys (decode_wide.cu)
TENSOR_CORE = [(*CONFIGS[1], dart.DEQUANT_PER_OP), (*CONFIGS[1], dart.DEQUANT_FUSED), (*CONFIGS[2], dart.DEQUANT_PER_OP),
               (torch.float16, dict(bits=8, key_group_size=128, value_group_size=64, promote_ratio=0.0), dart.DEQUANT_PER_OP)]


@pytest.mark.parametrize("dtype,cfg,flavour", TENSOR_CORE)
@pytest.mark.parametrize("pages", [1, 2, 4, 5, 6, 8, 12])
def test_a_page_of_nan_logits(dtype, cfg, flavour, pages, decode_split):
    # an Inf makes the scale of its channel infinite: every key of the page has a NaN (0 * Inf) there
    gen = torch.Generator().manual_seed(pages)
    keys, values = (torch.randn(1, 2, 32 + pages * 128 + 3, 128, generator=gen) for _ in range(2))
    query = torch.randn(1, 8, 1, 128, generator=gen).to(dtype).cuda()
    for page in range(pages):
        bad = keys.clone()
        bad[:, 1, 32 + 128 * page + 5, 9] = float("inf")
        cache = make(dtype, cfg, bad, values)
        for split in (None, "aligned", "unaligned"):
            decode_split(split)
            out = dart.fused_dart_attention(query, cache, flavour=flavour)
            assert out[:, 4:].isnan().all() and out[:, :4].isfinite().all(), (page, split)


@pytest.mark.parametrize("dtype,cfg,flavour", TENSOR_CORE)
@pytest.mark.parametrize("tokens", [[0, 16], [16, 32], [0, 32], [3, 4], [32 + 3 * 128, 32 + 3 * 128 + 3], [32 + 3 * 128 + 2, 32 + 3 * 128 + 3]])
def test_nan_keys_among_dense_tokens(dtype, cfg, flavour, tokens):
    gen = torch.Generator().manual_seed(4)
    keys, values = (torch.randn(1, 2, 32 + 3 * 128 + 3, 128, generator=gen) for _ in range(2))
    keys[:, 1, tokens[0]:tokens[1], 9] = float("nan")
    out = dart.fused_dart_attention(torch.randn(1, 8, 1, 128, generator=gen).to(dtype).cuda(), make(dtype, cfg, keys, values), flavour=flavour)
    assert out[:, 4:].isnan().all() and out[:, :4].isfinite().all()


@pytest.mark.parametrize("dtype,cfg,flavour", [TENSOR_CORE[0], TENSOR_CORE[2]])
def test_nan_keys_packed_before_their_values(dtype, cfg, flavour):
    # keys packed to the last page, the newest 128 values dense: those tokens go one to a warp
    gen = torch.Generator().manual_seed(5)
    tokens = 32 + 3 * 128
    keys, values = (torch.randn(1, 2, tokens + 40, 128, generator=gen) for _ in range(2))
    keys[:, 1, tokens - 1, 9] = float("inf")
    cache = dart.DartKVCache(dart.DartKVCacheConfig(page_size=128, sink_tokens=32, local_tokens=1, value_local_tokens=128,
                                                    metadata_dtype=torch.float16, **cfg))
    for start in range(0, tokens + 40, 64):
        cache.append(*(x[:, :, start:start + 64].to(dtype).cuda() for x in (keys, values)))
    out = dart.fused_dart_attention(torch.randn(1, 8, 1, 128, generator=gen).to(dtype).cuda(), cache, flavour=flavour)
    assert out[:, 4:].isnan().all() and out[:, :4].isfinite().all()


@pytest.mark.parametrize("dtype,cfg,flavour", [TENSOR_CORE[0], TENSOR_CORE[2], TENSOR_CORE[3]])
def test_infinitely_small_logits_of_dense_tokens_weigh_nothing(dtype, cfg, flavour):
    gen = torch.Generator().manual_seed(6)
    keys, values = (torch.randn(1, 1, 32 + 2 * 128 + 3, 128, generator=gen) for _ in range(2))
    query = (torch.rand(1, 2, 1, 128, generator=gen) + 0.5).to(dtype).cuda()
    keys[:, :, 16:32, 4] = float("-inf")    # a whole tile of sixteen tokens
    keys[:, :, -1, 4] = float("-inf")       # one token of another
    cache = make(dtype, cfg, keys, values)
    k, v = cache.get()
    ref = torch.softmax(query.double() @ k.double().transpose(2, 3) * 128 ** -0.5, -1) @ v.double()
    # fp32 sums of values up to 5, one rounding to the 16-bit type (half an ulp: at most 2^-8 or 2^-11 of the result)
    out = dart.fused_dart_attention(query, cache, flavour=flavour).double()
    assert torch.all((out - ref).abs() <= ref.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) + 2e-5)
