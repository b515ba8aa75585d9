"""More rows than the device holds blocks: memory that an earlier block of an SM used for its copies becomes merge buffers, and
the split of rows over blocks must not show in the result."""

import pytest
import torch

import dartkv_b200 as dart

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens", [32 + 8 * 128 + 77, 32 + 9 * 128, 32 + 21 * 128 + 1])
@pytest.mark.parametrize("flavour", [dart.DEQUANT_PER_OP, dart.DEQUANT_FUSED])
def test_many_rows(dtype, tokens, flavour, decode_split):
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    cache = dart.DartKVCache(dart.DartKVCacheConfig(bits=2, page_size=128, key_group_size=128, value_group_size=64, sink_tokens=32,
                                                    hold_partial_pages=True, promote_ratio=0.25, metadata_dtype=dtype))
    cache.append(*(torch.randn(70, 8, tokens, 128, generator=gen, device="cuda", dtype=dtype) for _ in range(2)))
    for rep in (2, 4):
        query = torch.randn(70, 8 * rep, 1, 128, generator=gen, device="cuda", dtype=dtype)
        first = None
        for split in ("aligned", "unaligned", "unaligned:37", None):
            decode_split(split)
            for _ in range(3):
                out = dart.fused_dart_attention(query, cache, flavour=flavour, fallback=False).float()
                assert cache.decode_status() == 0
                first = out if first is None else first
                # two roundings of fp32 results that differ by the order of their sums: an ulp.  The unrounded flavour also rounds
                # its weights p * scale to fp16 after a scaling that depends on the pages a warp has seen: 2^-11 of values below 6, twice.
                bound = first.abs() * (2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10) + (6e-3 if flavour == dart.DEQUANT_FUSED else 4e-5)
                assert torch.all((out - first).abs() <= bound), float((out - first).abs().max())
