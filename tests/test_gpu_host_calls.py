"""Calls that go through the native host path against the same calls with strided tensors and in forms that it leaves to Python, and errors
that stay what they were."""

import pytest
import torch

import dartkv_b200 as dart

pytestmark = pytest.mark.gpu


def randn(*shape, dtype=torch.float16):
    return torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(len(shape)), device="cuda").to(dtype)


@pytest.mark.parametrize("axis", [-1, -2, 1, 3])
@pytest.mark.parametrize("metadata", [None, torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_quantize_and_back(axis, metadata, dtype):
    data = randn(2, 3, 40, 64, dtype=dtype)
    call = dict(bits=4, group_size=8, metadata_dtype=metadata, axis=axis)
    ours, strided = dart.quantize(data, **call), dart.quantize(data.transpose(2, 3).contiguous().transpose(2, 3), **call)
    for name in ("values", "scale", "zero_point"):
        assert torch.equal(getattr(ours, name), getattr(strided, name))
    assert ours.axis == strided.axis == axis % 4 and ours.original_shape == (2, 3, 40, 64) and ours.scale.dtype == (metadata or dtype)
    assert (ours.original_dim, ours.padded_dim, ours.packed_dim, ours.groups) == (strided.original_dim, strided.padded_dim, strided.packed_dim, strided.groups)
    back = ours.dequantize()
    for name in ("values", "scale", "zero_point"):
        setattr(ours, name, torch.stack((getattr(ours, name),) * 2, -1)[..., 0])
        assert not getattr(ours, name).is_contiguous() and torch.equal(ours.dequantize(), back)
    ours.original_shape = list(ours.original_shape)                         # not a tuple: restored through Python
    assert torch.equal(ours.dequantize(), back)
    assert ours.dequantize(dtype=torch.bfloat16).dtype == torch.bfloat16


def test_mixed_keys_and_back():
    keys = randn(2, 3, 64, 32)
    ours, strided = (dart.quantize_key_mixed(k, group_size=32) for k in (keys, keys.transpose(1, 2).contiguous().transpose(1, 2)))
    for name in ("low_values", "high_values", "channel_indices", "scale", "zero_point"):
        assert torch.equal(getattr(ours, name), getattr(strided, name))
    back = ours.dequantize()
    for name in ("low_values", "high_values", "channel_indices", "scale", "zero_point"):
        setattr(ours, name, torch.stack((getattr(ours, name),) * 2, -1)[..., 0])
        assert not getattr(ours, name).is_contiguous() and torch.equal(ours.dequantize(), back)
    ours.channel_indices = ours.channel_indices.long()                      # restored through Python
    assert torch.equal(ours.dequantize(), back)


def test_strided_tensors_cross_into_native_code_once(monkeypatch):
    data = randn(2, 3, 64, 32).transpose(1, 2).contiguous().transpose(1, 2)
    packed, mixed = dart.quantize(data), dart.quantize_key_mixed(data, group_size=32)
    packed.values, mixed.low_values = (torch.stack((t, t), -1)[..., 0] for t in (packed.values, mixed.low_values))
    crossed = []

    class Host:
        def __getattr__(self, name):
            def call(*args):
                crossed.append(name)
                return getattr(host, name)(*args)
            return call

    host = dart._lib.HOST
    monkeypatch.setattr(dart._lib, "HOST", Host())
    monkeypatch.setattr(dart.quantization, "LIB", None)                     # nothing is left to do through ctypes
    monkeypatch.setattr(dart.mixed, "LIB", None)
    for call in (lambda: dart.quantize(data), lambda: dart.quantize_key_mixed(data, group_size=32), packed.dequantize, mixed.dequantize):
        call()
    assert crossed == ["quantize", "quantize_mixed", "dequantize", "dequantize_mixed"]


@pytest.mark.parametrize("call,error,text", [
    (dict(bits=3), ValueError, "bits must be one of"), (dict(group_size=0), ValueError, "positive integer"), (dict(group_size=2.5), ValueError, "positive integer"),
    (dict(axis=4), ValueError, "axis must be in"), (dict(axis=1.0), ValueError, "axis must be in"), (dict(division="other"), ValueError, "division"),
    (dict(metadata_dtype=torch.float64), TypeError, "float64"), (dict(metadata_dtype=torch.int32), TypeError, "floating point")])
def test_refused_quantizer_arguments(call, error, text):
    with pytest.raises(error, match=text):
        dart.quantize(randn(2, 3, 40, 64), **call)


def test_refused_data():
    data = randn(2, 3, 40, 64)
    data[1, 2, 3, 4] = float("nan")
    for call in (dart.quantize, dart.quantize_key_mixed):
        with pytest.raises(ValueError, match="finite"):
            call(data, group_size=8)
        call(data, group_size=8, check_finite=False)
    with pytest.raises(TypeError):
        dart.quantize(data.int())
    with pytest.raises(ValueError):
        dart.quantize(data[..., :0])
    with pytest.raises(RuntimeError, match="CUDA"):
        dart.quantize(data.cpu())


def test_pools_of_a_new_cache():
    config = dart.DartKVCacheConfig(bits=2, sink_tokens=3, page_size=128, key_group_size=128, hold_partial_pages=True)
    dirty = torch.full((1 << 22,), 255, dtype=torch.uint8, device="cuda")
    del dirty                                                                 # the allocator hands this memory out again
    cache = dart.DartKVCache(config)
    keys, values = randn(1, 2, 300, 128), randn(1, 2, 300, 128)
    cache.append(keys[:, :, :2], values[:, :, :2])
    cache.check_finite()
    spans = sorted((p.data_ptr(), p.data_ptr() + p.numel() * p.element_size()) for p in cache._pools.values())
    assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:]))
    assert all(p.data_ptr() % 256 == 0 for p in cache._pools.values())
    for start in range(2, 300, 75):                                           # the pools grow on the way
        cache.append(keys[:, :, start:start + 75], values[:, :, start:start + 75])
    whole = dart.DartKVCache(config, max_tokens=2000)
    whole.append(keys[:, :, :2], values[:, :, :2])
    for start in range(2, 300, 75):
        whole.append(keys[:, :, start:start + 75], values[:, :, start:start + 75])
    assert all(torch.equal(a, b) for a, b in zip(cache.get(), whole.get()))
    with torch.inference_mode():
        assert all(torch.equal(a, b) for a, b in zip(dart.DartKVCache(config).update(keys, values), whole.get()))
