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
