"""Materialization through the C entry points: outputs at any element-aligned address."""

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
