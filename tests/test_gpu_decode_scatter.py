"""The entry point that delivers rows to peers, as a world of one rank: every kernel's rows are bit for bit those of the call
without peers, in the caller's tensor and in the gathered one."""

import ctypes
import math

import pytest
import torch

import dartkv_b200 as dart
from dartkv_b200 import _lib
from dartkv_b200._lib import LIB, check, ptr, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,cfg", [(torch.float32, dict(bits=2, key_group_size=32, value_group_size=32)),
                                       (torch.float32, dict(bits=2, key_group_size=32, value_group_size=32, promote_ratio=0.25)),
                                       (torch.bfloat16, dict(bits=2, key_group_size=128, value_group_size=64, promote_ratio=0.25)),
                                       (torch.float16, dict(bits=4, key_group_size=128, value_group_size=64))])
@pytest.mark.parametrize("tokens", [1, 33, 160, 256, 257, 700])
def test_rows_equal_the_call_without_peers(dtype, cfg, tokens):
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    batch, heads, rep, dim = 2, 2, 3, 128
    cache = dart.DartKVCache(dart.DartKVCacheConfig(page_size=128, sink_tokens=2, hold_partial_pages=True, metadata_dtype=torch.float16, **cfg))
    cache.append(*(torch.randn(batch, heads, tokens, dim, generator=gen, device="cuda", dtype=dtype) for _ in range(2)))
    query = torch.randn(batch, heads * rep, dim, generator=gen, device="cuda", dtype=dtype)
    local = dart.decode_attention(query, cache)
    gathered = torch.full((batch + 1, heads * rep + 2, dim), 7.0, device="cuda", dtype=dtype)   # rows 1.., heads 2.. are this rank's
    flags = torch.zeros(4, dtype=torch.int32, device="cuda")
    peers = _lib.PeerScatter()
    peers.world_size, peers.rank, peers.epoch = 1, 0, 1
    peers.dst_row_begin, peers.dst_head_begin, peers.dst_heads_total = 1, 2, heads * rep + 2
    peers.out[0], peers.flags[0] = gathered.data_ptr(), flags.data_ptr()
    out = torch.empty_like(query)
    workspace, _ = cache.decode_workspace(heads * rep)
    check(LIB.dartkv_decode_attention_scatter(ctypes.byref(cache.descriptor), ptr(query), _lib.DTYPE_CODE[dtype], heads * rep,
                                              1.0 / math.sqrt(dim), dart.DEQUANT_PER_OP, tokens, ptr(workspace), workspace.numel(),
                                              ptr(out), ctypes.byref(peers), stream_ptr(query.device)))
    assert cache.decode_status() == 0
    assert torch.equal(out, local) and torch.equal(gathered[1:, 2:], local)
    gathered[1:, 2:] = 7.0
    assert torch.all(gathered == 7.0)
