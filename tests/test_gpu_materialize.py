"""Materialization: outputs at any element-aligned address, and ranges longer than one launch covers."""

import ctypes

import pytest
import torch

import dartkv_b200 as dart
from dartkv_b200 import _lib

pytestmark = pytest.mark.gpu


def build(dtype, tokens, heads=2, head_dim=64, seed=3, **cfg):
    gen = torch.Generator().manual_seed(seed)
    keys, values = (torch.randn(1, heads, tokens, head_dim, generator=gen).to(dtype).cuda() for _ in range(2))
    base = dict(bits=2, page_size=128, key_group_size=128, value_group_size=32, sink_tokens=5, promote_ratio=0.25)
    base.update(cfg)
    cache = dart.DartKVCache(dart.DartKVCacheConfig(**base))
    cache.append(keys, values)
    return cache


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("offset", [1, 2, 3, 8])
def test_output_at_an_element_offset(dtype, offset):
    cache = build(dtype, 5 + 2 * 128 + 9)
    keys, values = cache.get()
    n = keys.numel()
    stream = torch.cuda.current_stream().cuda_stream
    for out_dtype in (dtype, torch.float32):
        room = torch.zeros(2, n + 16, dtype=out_dtype, device="cuda")
        out = [room[i, offset:offset + n] for i in range(2)]
        desc = ctypes.byref(cache.descriptor)
        code = _lib.DTYPE_CODE[out_dtype]
        _lib.check(_lib.LIB.dartkv_cache_materialize_both(desc, 0, cache.seen_tokens, _lib.DEQUANT_PER_OP, out[0].data_ptr(),
                                                          out[1].data_ptr(), code, stream))
        assert torch.equal(out[0].view_as(keys), keys.to(out_dtype)) and torch.equal(out[1].view_as(values), values.to(out_dtype))
        room.zero_()
        for side in (0, 1):
            _lib.check(_lib.LIB.dartkv_cache_materialize(desc, side, 0, cache.seen_tokens, _lib.DEQUANT_PER_OP,
                                                         out[side].data_ptr(), code, stream))
        assert torch.equal(out[0].view_as(keys), keys.to(out_dtype)) and torch.equal(out[1].view_as(values), values.to(out_dtype))
        assert room[:, :offset].count_nonzero() == 0 and room[:, offset + n:].count_nonzero() == 0


@pytest.mark.parametrize("dtype,cfg", [(torch.float32, dict(bits=2)), (torch.bfloat16, dict(bits=8, hold_partial_pages=True))])
def test_ranges_longer_than_one_launch(dtype, cfg):
    # 65,535 tiles of 32 tokens on the general kernel, 65,535 spans of 128 tokens on the other one
    page = 128 * 65535 if dtype != torch.float32 else 32 * 65535
    cache = dart.DartKVCache(dart.DartKVCacheConfig(page_size=128, key_group_size=128, value_group_size=8, sink_tokens=5, **cfg),
                             max_tokens=page + 1000)
    gen = torch.Generator().manual_seed(1)
    piece = 65408
    keys, values = (torch.randn(1, 1, piece, 8, generator=gen).to(dtype).cuda() for _ in range(2))
    while cache.seen_tokens < page + 300:
        take = min(piece, page + 300 - cache.seen_tokens)
        cache.append(keys[:, :, :take], values[:, :, :take])
    for whole, side in zip(cache.get(), (0, 1)):
        for first, last in ((0, 700), (page - 400, page + 300), (page // 2, page // 2 + 500)):
            assert torch.equal(whole[:, :, first:last], cache._materialize(side, first, last))
