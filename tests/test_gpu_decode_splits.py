"""Work splits of the 2-bit kernels in units of four and of eight pages: odd and even counts of either, shares that end inside a row,
left padding that leaves a row's first units empty, against attention in 64 bits over the materialized cache."""

import pytest
import torch

import dartkv_b200 as dart

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,pages", [(2, 8), (2, 9), (3, 17), (5, 31), (7, 33), (37, 12), (41, 15), (2, 130)])
def test_units_of_pages(batch, pages, decode_split):
    gen = torch.Generator(device="cuda").manual_seed(pages)
    tokens = 32 + 128 * pages + 70
    cache = dart.DartKVCache(dart.DartKVCacheConfig(bits=2, page_size=128, key_group_size=128, value_group_size=64, sink_tokens=32,
                                                    hold_partial_pages=True, promote_ratio=0.25, metadata_dtype=torch.bfloat16))
    cache.append(*(torch.randn(batch, 2, tokens, 128, generator=gen, device="cuda", dtype=torch.bfloat16) for _ in range(2)))
    query = torch.randn(batch, 8, 1, 128, generator=gen, device="cuda", dtype=torch.bfloat16)
    k, v = (t.double() for t in cache.get())
    logits = query.double().view(batch, 2, 4, 128) @ k.transpose(2, 3) * 128 ** -0.5
    starts = torch.tensor([(b * 1531) % (tokens - 1) for b in range(batch)], dtype=torch.int32, device="cuda")
    for start in (None, starts):
        masked = logits if start is None else logits.masked_fill(torch.arange(tokens, device="cuda") < start.view(batch, 1, 1, 1), float("-inf"))
        ref = (torch.softmax(masked, -1) @ v).view(query.shape)
        fp32 = dart.fused_dart_attention(query.float(), cache, row_start=start, flavour=dart.DEQUANT_FUSED).double()
        for split in (None, "aligned", "unaligned", "unaligned:5", "unaligned:3"):
            decode_split(split)
            out = dart.fused_dart_attention(query, cache, row_start=start).double()
            # fp32 sums of values up to 5 and a rounding of the result, at most 2^-8 of it
            assert torch.all((out - ref).abs() <= ref.abs() * 2.0 ** -8 + 4e-5), (split, float((out - ref).abs().max()))
            out = dart.fused_dart_attention(query, cache, row_start=start, flavour=dart.DEQUANT_FUSED).double()
            # besides, weights q * scale and p * scale rounded to fp16: 2^-11 of three scales, some 6, in a result
            assert torch.all((out - fp32).abs() <= fp32.abs() * 2.0 ** -8 + 1.5e-2), (split, float((out - fp32).abs().max()))
        assert cache.decode_status() == 0
