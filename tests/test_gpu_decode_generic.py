"""The CUDA-core decode kernel cut into many splits (more than the merge keeps in registers), with head dimensions that do
not divide its blocks, against attention in 64 bits over the materialized cache."""

import pytest
import torch

import dartkv_b200 as dart

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("head_dim", [24, 40, 96, 128, 200, 256])
@pytest.mark.parametrize("tokens", [17 * 32, 17 * 32 + 1, 3000])
@pytest.mark.parametrize("hold", [True, False])
def test_many_splits(head_dim, tokens, hold):
    gen = torch.Generator().manual_seed(head_dim + tokens)
    keys, values = (torch.randn(2, 1, tokens, head_dim, generator=gen).cuda() for _ in range(2))
    cache = dart.DartKVCache(dart.DartKVCacheConfig(bits=2, page_size=128, key_group_size=32, value_group_size=8, sink_tokens=5,
                                                    hold_partial_pages=hold, promote_ratio=0.25 if head_dim == 40 else 0.0))
    cache.append(keys[:, :, :tokens // 2], values[:, :, :tokens // 2])
    cache.append(keys[:, :, tokens // 2:], values[:, :, tokens // 2:])
    k, v = (t.double() for t in cache.get())
    row_start = torch.tensor([0, tokens // 3], dtype=torch.int32, device="cuda")
    for rep in (1, 3, 5, 16):
        query = torch.randn(2, rep, 1, head_dim, generator=gen).cuda()
        logits = query.double() @ k.transpose(2, 3) * head_dim ** -0.5
        for start in (None, row_start):
            if start is not None:
                logits = logits.masked_fill(torch.arange(tokens, device="cuda") < start.view(2, 1, 1, 1), float("-inf"))
            out = dart.fused_dart_attention(query, cache, row_start=start)
            # fp32 sums over at most 3,000 weights that add up to one, of values up to 5: 1e-5 as for the other fp32 checks
            assert (out.double() - torch.softmax(logits, -1) @ v).abs().max() < 1e-5
