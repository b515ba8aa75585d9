"""A workspace that begins at any multiple of four bytes, on every kernel that writes partials, gives the bits of one that begins at a
multiple of eight, and is not written past its size."""

import ctypes

import pytest
import torch

import dartkv_b200 as dart
from dartkv_b200 import _lib
from dartkv_b200._lib import LIB, check, ptr, stream_ptr

pytestmark = pytest.mark.gpu


def build(batch, tokens, dtype, seed=0, **cfg):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    base = dict(bits=2, page_size=128, key_group_size=128, value_group_size=64, sink_tokens=32, hold_partial_pages=True, metadata_dtype=dtype)
    base.update(cfg)
    cache = dart.DartKVCache(dart.DartKVCacheConfig(**base))
    cache.append(*(torch.randn(batch, 2, tokens, 128, generator=gen, device="cuda", dtype=dtype) for _ in range(2)))
    return cache


@pytest.mark.parametrize("batch,tokens,rep,flavour,dtype,cfg", [
    (2, 800, 4, dart.DEQUANT_PER_OP, torch.bfloat16, dict(promote_ratio=0.25)),        # two warps a page, warp-per-row merge
    (2, 9000, 3, dart.DEQUANT_PER_OP, torch.float16, dict(promote_ratio=0.25)),        # more slots than that merge takes
    (2, 9000, 4, dart.DEQUANT_FUSED, torch.bfloat16, dict(promote_ratio=0.25)),
    (2, 3000, 4, dart.DEQUANT_PER_OP, torch.float16, dict(bits=4)),
    (2, 3000, 4, dart.DEQUANT_PER_OP, torch.float16, dict(bits=8)),
    (2, 3000, 8, dart.DEQUANT_PER_OP, torch.bfloat16, dict(promote_ratio=0.25)),
    (16, 2200, 20, dart.DEQUANT_PER_OP, torch.bfloat16, dict(promote_ratio=0.25)),     # a page restored once for all rows
    (2, 700, 4, dart.DEQUANT_PER_OP, torch.float32, dict()),
    (2, 3000, 4, dart.DEQUANT_PER_OP, torch.float32, dict(promote_ratio=0.25)),
])
def test_workspaces_that_begin_between_two_multiples_of_eight(batch, tokens, rep, flavour, dtype, cfg):
    cache = build(batch, tokens, dtype, **cfg)
    gen = torch.Generator(device="cuda").manual_seed(1)
    query = torch.randn(batch, 2 * rep, 128, generator=gen, device="cuda", dtype=dtype)
    nbytes = LIB.dartkv_decode_workspace_bytes(ctypes.byref(cache.descriptor), 2 * rep, tokens)
    outs = []
    for offset in (0, 4, 8, 12):
        buffer = torch.zeros(nbytes + 64, dtype=torch.uint8, device="cuda")
        assert buffer.data_ptr() % 16 == 0
        buffer[offset + nbytes:] = 77
        out = torch.empty_like(query)
        check(LIB.dartkv_decode_attention_rows(ctypes.byref(cache.descriptor), ptr(query), _lib.DTYPE_CODE[dtype], 2 * rep, 128 ** -0.5, flavour,
                                               tokens, None, buffer.data_ptr() + offset, nbytes, ptr(out), stream_ptr(query.device)))
        assert int(buffer[offset:offset + 4].sum()) == 0 and torch.all(buffer[offset + nbytes:] == 77)
        outs.append(out)
    assert all(torch.equal(outs[0], out) for out in outs[1:])
