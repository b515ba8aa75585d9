"""What the native host path leaves to the Python code, and what it keeps between calls."""

import pytest
import torch

import dartkv_b200 as dart
from dartkv_b200 import _lib
from dartkv_b200.synthetic import make_kvq

pytestmark = pytest.mark.gpu


def build(tokens=32 + 3 * 128 + 5, batch=2, heads=2, dtype=torch.bfloat16, seed=1, max_tokens=None, **cfg):
    keys, values, _ = make_kvq(seed, batch, heads, tokens + 1, 128, query_heads=heads, dtype=dtype, outlier_fraction=0.05)
    base = dict(bits=2, page_size=128, key_group_size=128, value_group_size=64, sink_tokens=32, hold_partial_pages=True,
                promote_ratio=0.25, metadata_dtype=dtype)
    base.update(cfg)
    cache = dart.DartKVCache(dart.DartKVCacheConfig(**base), max_tokens=max_tokens)
    keys, values = keys.cuda(), values.cuda()
    cache.append(keys[:, :, :tokens], values[:, :, :tokens])
    return cache, keys[:, :, tokens:], values[:, :, tokens:]


def test_tensors_on_another_device_than_the_pools_are_left_to_the_checks():
    # a second GPU is not needed: the binding is told that the pools are on one
    cache, keys, values = build()
    query = torch.randn(2, 8, 1, 128, device="cuda", dtype=torch.bfloat16)
    dart.fused_dart_attention(query, cache)
    state = [getattr(cache._c_state, name) for name, _ in cache._c_state._fields_]
    launches = _lib.LIB.dartkv_launch_count()
    *addresses, device = cache._append_args
    assert device == cache._device.index
    assert _lib.HOST.append(keys, values, *addresses, device + 1) == _lib.HOST.SLOW_PATH
    key = 8, torch.cuda.current_stream().cuda_stream
    arguments = cache._decode_args[key]
    assert _lib.HOST.decode(query, *arguments, cache.seen_tokens, 0.1, 0, None, device + 1) is None
    assert [getattr(cache._c_state, name) for name, _ in cache._c_state._fields_] == state
    # the public calls: the Python checks find the tensors on another device than the cache says
    cache._device = torch.device("cuda", device + 1)
    cache._bind_native()
    cache._decode_args[key] = arguments
    with pytest.raises(ValueError):
        cache.append(keys, values)
    with pytest.raises(ValueError):
        dart.fused_dart_attention(query, cache)
    with pytest.raises(ValueError):
        dart.decode_attention(query[:, :, 0], cache)
    assert _lib.LIB.dartkv_launch_count() == launches


@pytest.mark.parametrize("rep", [1, 4, 5])
@pytest.mark.parametrize("flavour", [dart.DEQUANT_PER_OP, dart.DEQUANT_FUSED])
def test_a_query_from_an_odd_element_on(flavour, rep):
    cache, _, _ = build(tokens=32 + 9 * 128 + 5)
    query = torch.randn(2, 2 * rep, 1, 128, device="cuda").bfloat16()
    ref = dart.fused_dart_attention(query, cache, flavour=flavour)
    odd = torch.empty(query.numel() + 1, device="cuda", dtype=query.dtype)[1:].view(query.shape)
    odd.copy_(query)
    assert odd.data_ptr() % 4 == 2
    for call in range(2):       # the native path, then the Python one
        if call:
            cache._decode_args = {}
        assert torch.equal(dart.fused_dart_attention(odd, cache, flavour=flavour), ref)


def test_one_step_of_more_pages_than_a_shared_grid_holds():
    # the C entry point takes chunks that the Python side would cut: 32,768 pages, each of them the same tokens
    import ctypes

    pages = 32768
    gen = torch.Generator().manual_seed(4)
    keys, values = (torch.randn(1, 1, 1, 128, generator=gen).bfloat16().cuda() for _ in range(2))
    cache = dart.DartKVCache(dart.DartKVCacheConfig(bits=2, page_size=128, key_group_size=128, value_group_size=64, sink_tokens=0,
                                                    hold_partial_pages=True, promote_ratio=0.25), max_tokens=(pages + 1) * 128)
    cache.append(keys.expand(-1, -1, 128, -1), values.expand(-1, -1, 128, -1))
    _lib.check(_lib.LIB.dartkv_cache_append_step(
        ctypes.byref(cache.descriptor), ctypes.byref(cache._c_cfg), ctypes.byref(cache._c_state), keys.data_ptr(), values.data_ptr(),
        pages * 128, 0, 0, 0, None, cache._pools["nonfinite"].data_ptr(), ctypes.byref(cache._plan),
        torch.cuda.current_stream().cuda_stream))
    assert cache._pools["state"][:4].tolist() == [(pages + 1) * 128, pages + 1] + [(pages + 1) * 128] * 2
    for name, rows in (("k_pages", pages + 1), ("v_codes", (pages + 1) * 128), ("v_meta", (pages + 1) * 128)):
        pool = cache._pools[name][0, 0, :rows].flatten(1)
        assert torch.equal(pool, pool[:1].expand_as(pool))


def test_calls_that_may_overlap_have_scratch_of_their_own():
    cache, _, _ = build(tokens=32 + 9 * 128 + 5)
    query = torch.randn(2, 2 * 16, 1, 128, device="cuda").bfloat16()
    reps = (1, 2, 3, 4, 5, 8, 9, 16)
    ref = {rep: dart.fused_dart_attention(query[:, :2 * rep], cache) for rep in reps}
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    ranges = {}
    for stream in streams:
        with torch.cuda.stream(stream):
            for rep in reps:
                assert torch.equal(dart.fused_dart_attention(query[:, :2 * rep], cache), ref[rep])
                buffer = cache.decode_workspace(2 * rep)[0]
                ranges[min(rep, 4) if rep <= 4 else 8 if rep <= 8 else 16, stream] = (buffer.data_ptr(), buffer.numel())
                # what the native path is given is that buffer
                assert cache._decode_args[2 * rep, stream.cuda_stream][1] == buffer.data_ptr()
    spans = sorted(ranges.values())
    assert len(spans) == 2 * 6 and all(a + n <= b for (a, n), (b, _) in zip(spans, spans[1:]))
    held = len(cache._scratch)
    for _ in range(3):          # nothing is made again
        for stream in streams:
            with torch.cuda.stream(stream):
                dart.fused_dart_attention(query[:, :8], cache)
    assert len(cache._scratch) == held and cache.decode_status() == 0


@pytest.mark.parametrize("before", [True, False])
def test_captured_calls_take_scratch_that_exists(before):
    cache, _, _ = build(max_tokens=4096)
    query = torch.randn(2, 8, 1, 128, device="cuda").bfloat16()
    other, _, _ = build()
    ref = dart.fused_dart_attention(query, other)      # kernel attributes are set outside the capture
    made = cache.decode_workspace(8)[0].data_ptr() if before else None
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        capturing = torch.cuda.current_stream().cuda_stream
        out = dart.fused_dart_attention(query, cache)
    assert len(cache._scratch) == 1 and (8, capturing) not in cache._decode_args
    for _ in range(2):
        out.zero_()
        graph.replay()
        assert torch.equal(out, ref)
    # an eager call does not take the graph's memory
    assert torch.equal(dart.fused_dart_attention(query, cache), ref)
    assert len(cache._scratch) == (1 if before else 2)
    if before:
        assert cache._scratch[0].data_ptr() == made


def test_the_first_call_on_a_cache_is_native():
    cache, keys, values = build()
    query = torch.randn(2, 8, 1, 128, device="cuda").bfloat16()
    for change in (lambda: None, lambda: cache.append(keys, values), lambda: cache.reorder_batch([1, 0]),
                   lambda: cache._ensure_capacity(2 * cache._desc.max_key_pages, cache._desc.max_value_tokens)):
        change()
        launches = _lib.LIB.dartkv_launch_count()
        first = cache.decode_native(query, None, _lib.DEQUANT_PER_OP, None)
        assert first is not None and _lib.LIB.dartkv_launch_count() == launches + 2
        assert torch.equal(cache.decode_native(query, None, _lib.DEQUANT_PER_OP, None), first)
        assert torch.equal(dart.decode_attention(query[:, :, 0], cache, out=torch.empty_like(first[:, :, 0])), first[:, :, 0])
    # calls that the Python code refuses or serves otherwise make no scratch
    made = len(cache._scratch)
    for odd in (query[:, :7], query[:1], query.cpu(), torch.randn(2, 2 * 40, 1, 128, device="cuda").bfloat16()):
        assert cache.decode_native(odd, None, _lib.DEQUANT_PER_OP, None) is None
    assert len(cache._scratch) <= made + 1


LAYOUTS = {"contiguous": lambda t: t.contiguous(), "projection": lambda t: t.transpose(1, 2).contiguous().transpose(1, 2),
           "wide_rows": lambda t: torch.cat([t, t], -1)[..., :128], "every_other": lambda t: torch.stack([t, -t], -1)[..., 0],
           "same_batch": lambda t: t[:1].contiguous().expand(t.shape[0], -1, -1, -1),
           "odd_start": lambda t: torch.cat([t.new_zeros(3), t.flatten()])[3:].view(t.shape)}


@pytest.mark.parametrize("keys_as", sorted(LAYOUTS))
@pytest.mark.parametrize("values_as", sorted(LAYOUTS))
def test_layouts_of_keys_and_values(keys_as, values_as):
    # whatever the strides of the two tensors, the pools get the bytes of contiguous ones
    gen = torch.Generator().manual_seed(6)
    base = torch.randn(2, 2, 2, 32 + 3 * 128 + 41, 128, generator=gen).bfloat16().cuda()
    base[:, 1] = base[:, :1].squeeze(1) if "same_batch" in (keys_as, values_as) else base[:, 1]
    caches = [dart.DartKVCache(dart.DartKVCacheConfig(bits=2, page_size=128, key_group_size=128, value_group_size=64, sink_tokens=32,
                                                      hold_partial_pages=True, promote_ratio=0.25, metadata_dtype=torch.bfloat16))
              for _ in range(2)]
    start = 0
    for chunk in (300, 1, 1, 40, 1, 114):
        keys, values = base[0, :, :, start:start + chunk], base[1, :, :, start:start + chunk]
        caches[0].append(keys.contiguous(), values.contiguous())
        caches[1].append(LAYOUTS[keys_as](keys), LAYOUTS[values_as](values))
        start += chunk
    assert start == base.shape[3]
    for (k0, v0), (k1, v1) in zip(*(cache.iter_segments() for cache in caches)):
        for a, b in ((k0, k1), (v0, v1)):
            names = ("values", "low_values", "high_values", "channel_indices", "scale", "zero_point")
            fields = [("", a, b)] if isinstance(a, torch.Tensor) else [(n, getattr(a, n), getattr(b, n)) for n in names if hasattr(a, n)]
            for name, x, y in fields:
                assert torch.equal(x, y), name
