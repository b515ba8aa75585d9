"""Device memory of a cache's pools: each is held by itself, so that replacing or dropping one gives its memory back."""

import pytest
import torch

import dartkv_b200 as dart

pytestmark = pytest.mark.gpu


def build(batch=16, tokens=600, **cfg):
    base = dict(bits=2, page_size=128, key_group_size=128, value_group_size=64, sink_tokens=32, hold_partial_pages=True, promote_ratio=0.25)
    base.update(cfg)
    cache = dart.DartKVCache(dart.DartKVCacheConfig(metadata_dtype=torch.bfloat16, **base), max_tokens=tokens)
    data = torch.randn(batch, 4, tokens, 128, device="cuda", dtype=torch.bfloat16)
    cache.append(data, data)
    return cache


def nbytes(tensor):
    return tensor.numel() * tensor.element_size()


def held(what="current"):
    """Bytes that live tensors asked for (the allocator's blocks may be larger)."""
    return torch.cuda.memory_stats()[f"requested_bytes.all.{what}"]


@pytest.mark.parametrize("cfg", [dict(), dict(value_bits=8, value_group_size=16)])
def test_a_reorder_gives_the_earlier_pools_back(cfg):
    cache = build(**cfg)
    indices = torch.arange(15, -1, -1, device="cuda")
    before, largest = held(), max(nbytes(p) for p in cache._pools.values())
    torch.cuda.reset_peak_memory_stats()
    cache.reorder_batch(indices)
    assert held() == before
    assert held("peak") <= before + largest + 4096     # one pool at a time, besides the checked indices
    rows = sum(nbytes(cache._pools[name]) for name in ("k_sink", "v_sink", "k_ring", "v_ring", "k_pages", "v_codes", "v_meta"))
    cache.reorder_batch(indices[:4])
    assert before - held() == rows - rows // 4


def test_a_kept_segment_holds_its_own_pool_only():
    start = held()
    cache = build()
    sink = cache.iter_segments()[0][0]
    assert sink.data_ptr() == cache._pools["k_sink"].data_ptr()
    size = nbytes(cache._pools["k_sink"])
    del cache
    assert held() - start == size
