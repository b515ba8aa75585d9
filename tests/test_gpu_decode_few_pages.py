"""Blocks of the 2-bit decode kernels with at most four pages of a row, whose warps share a page in twos, next to blocks and rows
with more, where a warp takes a page alone: one to thirteen pages, shares that run from row to row, rows whose left padding leaves
few pages.  The per-op flavour against attention in 64 bits over the materialized cache, the unrounded one against the CUDA-core
kernel, which computes it in fp32 throughout."""

import pytest
import torch

import dartkv_b200 as dart

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,metadata,promote,value_group", [(torch.bfloat16, torch.bfloat16, 0.25, 64), (torch.float16, torch.float16, 0.1, 128),
                                                                (torch.bfloat16, torch.float16, 0.0, 64)])
@pytest.mark.parametrize("pages", [1, 2, 3, 4, 5, 7, 8, 9, 12, 13])
def test_few_pages(dtype, metadata, promote, value_group, pages, decode_split):
    gen = torch.Generator(device="cuda").manual_seed(pages)
    tokens = 32 + 128 * pages + 5
    cache = dart.DartKVCache(dart.DartKVCacheConfig(bits=2, page_size=128, key_group_size=128, value_group_size=value_group, sink_tokens=32,
                                                    hold_partial_pages=True, promote_ratio=promote, metadata_dtype=metadata))
    cache.append(*(torch.randn(3, 2, tokens, 128, generator=gen, device="cuda", dtype=dtype) for _ in range(2)))
    query = torch.randn(3, 8, 1, 128, generator=gen, device="cuda", dtype=dtype)
    k, v = (t.double() for t in cache.get())
    logits = (query.double().view(3, 2, 4, 128) @ k.transpose(2, 3)) * 128 ** -0.5
    # a page in the middle cut by the row's start, four pages and a bit left, one token left
    pads = torch.tensor([max(0, tokens // 2 - 40), max(0, tokens - 5 - 4 * 128 - 1), tokens - 1], dtype=torch.int32, device="cuda")
    half_ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11   # of a result: at most this share of it
    for start in (None, pads):
        masked = logits if start is None else logits.masked_fill(torch.arange(tokens, device="cuda") < start.view(3, 1, 1, 1), float("-inf"))
        weights = torch.softmax(masked, -1)
        ref = (weights @ v).view(query.shape)
        spread = (weights @ v.abs()).view(query.shape)
        fp32 = dart.fused_dart_attention(query.float(), cache, row_start=start, flavour=dart.DEQUANT_FUSED).double()
        for split in (None, "aligned", "unaligned", "unaligned:5", "unaligned:4", "unaligned:1"):
            decode_split(split)
            out = dart.fused_dart_attention(query, cache, row_start=start, flavour=dart.DEQUANT_PER_OP).double()
            # fp32 sums of values up to 5 and a rounding of the result
            assert torch.all((out - ref).abs() <= ref.abs() * half_ulp + 4e-5), (split, float((out - ref).abs().max()))
            out = dart.fused_dart_attention(query, cache, row_start=start, flavour=dart.DEQUANT_FUSED).double()
            # besides, weights rounded to fp16 (half an ulp: 2^-11): p * scale, which moves a result by 2^-11 of scale * code, of
            # three scales, some 6; and q * scale, each an error of its own sign, some 2^-11 * |scale code| <= 2^-9 * 128^0.5 *
            # 128^-0.5 in a logit and as much of every weight
            assert torch.all((out - fp32).abs() <= fp32.abs() * half_ulp + 3e-3 + spread * 2.0 ** -9), (split, float((out - fp32).abs().max()))
        assert cache.decode_status() == 0
