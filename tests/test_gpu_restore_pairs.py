"""Restored values with two codes per register: every code width and dtype pair, scales from subnormal to beyond what a packed
multiply-add could take, infinite ones too, partial words at the end, against the elementwise definition."""

import pytest
import torch

import dartkv_b200 as dart
from dartkv_b200 import _lib

pytestmark = pytest.mark.gpu
DTYPES = [torch.float16, torch.bfloat16]


def expected(codes, scale, zero, out, flavour):
    if flavour == _lib.DEQUANT_PER_OP:                     # each step rounded to the metadata dtype, then the cast
        return (codes.to(scale.dtype) * scale + zero).to(out)
    wide = codes.double() * scale.double() + zero.double() # one fp32 multiply-add: exact here but for its own rounding
    return wide.float().to(out)


def metadata(shape, dtype, gen):
    scale = torch.rand(shape, generator=gen, device="cuda") + 0.5
    scale *= 2.0 ** torch.randint(-20, 15, shape, generator=gen, device="cuda")
    scale.view(-1)[::37] = float("inf")
    return scale.to(dtype), (torch.randn(shape, generator=gen, device="cuda") * 100).to(dtype)


@pytest.mark.parametrize("md", DTYPES)
@pytest.mark.parametrize("out", DTYPES)
@pytest.mark.parametrize("flavour", [_lib.DEQUANT_PER_OP, _lib.DEQUANT_FP32])
@pytest.mark.parametrize("bits", [2, 4, 8])
@pytest.mark.parametrize("axis,shape,group", [(-1, (3, 5, 128), 32), (-2, (3, 77, 10), 32), (-2, (2, 128, 128), 64)])
def test_functional(md, out, flavour, bits, axis, shape, group):
    gen = torch.Generator(device="cuda").manual_seed(bits)
    data = torch.randn(shape, generator=gen, device="cuda").to(out)
    packed = dart.quantize(data, bits=bits, group_size=group, metadata_dtype=md, axis=axis)
    packed.scale, packed.zero_point = metadata(packed.scale.shape, md, gen)
    got = packed.dequantize(flavour=flavour)
    codes = dart.quantization._unpack(packed.values, bits, packed.packed_dim)[..., : packed.original_dim]
    scale, zero = (m.repeat_interleave(group, -1)[..., : packed.original_dim] for m in (packed.scale, packed.zero_point))
    ref = expected(codes, scale, zero, out, flavour).movedim(-1, axis)
    assert torch.equal(got.isnan(), ref.isnan()) and torch.equal(got.nan_to_num(7.0), ref.nan_to_num(7.0))


@pytest.mark.parametrize("md", DTYPES)
@pytest.mark.parametrize("out", DTYPES)
@pytest.mark.parametrize("tokens,group", [(128, 128), (77, 32)])
def test_promoted_channels(md, out, tokens, group):
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    keys = torch.randn(2, 3, tokens, 128, generator=gen, device="cuda").to(out)
    packed = dart.quantize_key_mixed(keys, group_size=group, promote_ratio=0.3, metadata_dtype=md)
    packed.scale, packed.zero_point = metadata(packed.scale.shape, md, gen)
    codes = dart.quantization._unpack(packed.low_values, 2, group).flatten(3)[..., :tokens]
    high = dart.quantization._unpack(packed.high_values, 2, group).flatten(3)[..., :tokens]
    index = packed.channel_indices.long()[..., None].expand(-1, -1, -1, tokens)
    codes = codes.int().scatter_add(2, index, 4 * high.int())
    scale, zero = (m.repeat_interleave(group, -1)[..., :tokens] for m in (packed.scale, packed.zero_point))
    for flavour in (_lib.DEQUANT_PER_OP, _lib.DEQUANT_FP32):
        got, ref = packed.dequantize(flavour=flavour), expected(codes, scale, zero, out, flavour).transpose(2, 3)
        assert torch.equal(got.isnan(), ref.isnan()) and torch.equal(got.nan_to_num(7.0), ref.nan_to_num(7.0))


@pytest.mark.parametrize("dtype,md", [(torch.float16, torch.float16), (torch.bfloat16, torch.float16), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("key_bits,value_bits,promote", [(2, 2, 0.25), (4, 8, 0.0), (8, 4, 0.0)])
def test_cache_contents_with_large_scales(dtype, md, key_bits, value_bits, promote):
    gen = torch.Generator(device="cuda").manual_seed(5)
    cache = dart.DartKVCache(dart.DartKVCacheConfig(key_bits=key_bits, value_bits=value_bits, page_size=128, key_group_size=128, value_group_size=64,
                                                    sink_tokens=5, hold_partial_pages=True, promote_ratio=promote, metadata_dtype=md))
    keys, values = (((torch.rand(2, 2, 300, 128, generator=gen, device="cuda") - 0.5) * 60000).to(dtype) for _ in range(2))
    cache.append(keys, values)
    got = cache.get()
    for side in range(2):
        parts = []
        for segment in (pair[side] for pair in cache.iter_segments()):
            parts.append(segment if isinstance(segment, torch.Tensor) else segment.dequantize())
        assert torch.equal(got[side], torch.cat(parts, dim=2)) and got[side].isfinite().all()
