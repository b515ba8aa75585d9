"""More rows than the device holds blocks: memory that an earlier block of an SM used for its copies becomes merge buffers, and
the split of rows over blocks must not show in the result."""

import pytest
import torch

import dartkv_b200 as dart

pytestmark = pytest.mark.gpu

ROWS = [0, 1, 34, 35, 68, 69]   # of the batch, compared with attention in 64 bits


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens", [32 + 8 * 128 + 77, 32 + 9 * 128, 32 + 21 * 128 + 1])
@pytest.mark.parametrize("flavour", [dart.DEQUANT_PER_OP, dart.DEQUANT_FUSED])
def test_many_rows(dtype, tokens, flavour, decode_split):
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    cache = dart.DartKVCache(dart.DartKVCacheConfig(bits=2, page_size=128, key_group_size=128, value_group_size=64, sink_tokens=32,
                                                    hold_partial_pages=True, promote_ratio=0.25, metadata_dtype=dtype))
    cache.append(*(torch.randn(70, 8, tokens, 128, generator=gen, device="cuda", dtype=dtype) for _ in range(2)))
    k, v = (t[ROWS].double() for t in cache.get())
    half_ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11   # of a result: at most this share of it
    # fp32 sums besides; the unrounded flavour's weights p * scale are rounded to fp16, 2^-11 of scale * code, some 6, with a sign of
    # its own for each of over 1,000 tokens that weigh at most a tenth together with their neighbours
    absolute = 1e-3 if flavour == dart.DEQUANT_FUSED else 4e-5
    for rep in (2, 4):
        query = torch.randn(70, 8 * rep, 1, 128, generator=gen, device="cuda", dtype=dtype)
        if flavour == dart.DEQUANT_PER_OP:
            logits = query[ROWS].double().view(len(ROWS), 8, rep, 128) @ k.transpose(2, 3) * 128 ** -0.5
            ref = (torch.softmax(logits, -1) @ v).view(len(ROWS), 8 * rep, 1, 128)
        else:   # what the CUDA-core kernel computes in fp32 throughout
            ref = dart.fused_dart_attention(query.float(), cache, flavour=flavour)[ROWS].double()
        first = None
        for split in ("aligned", "unaligned", "unaligned:37", None):
            decode_split(split)
            for _ in range(3):
                out = dart.fused_dart_attention(query, cache, flavour=flavour, fallback=False)
                assert cache.decode_status() == 0
                first = out.float() if first is None else first
                # two roundings of results that differ by the order of their sums, and by their maxima the unrounded one's weights
                assert torch.all((out.float() - first).abs() <= first.abs() * 2 * half_ulp + absolute), float((out.float() - first).abs().max())
                off = (out[ROWS].double() - ref).abs()
                assert torch.all(off <= ref.abs() * half_ulp + absolute), (split, float(off.max()))
