"""Groups along the tokens that a thread of the column quantizer keeps in registers and those it reads twice, ragged last
groups, and channel selection by one block or by a cluster of blocks per row, against the same rules in torch."""

import numpy as np
import pytest
import torch

import dartkv_b200 as dart
from tests.helpers import to_np
from tests.test_gpu_quantize_nonfinite import expected, pack, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("bits", [2, 4, 8])
@pytest.mark.parametrize("group", [16, 32, 64, 96, 128, 256])
@pytest.mark.parametrize("tokens", [1, 31, 128, 129, 300])
def test_columns(dtype, bits, group, tokens):
    if group * bits % 32:
        return
    x = torch.randn(3, tokens, 70, generator=torch.Generator().manual_seed(group + tokens)).to(dtype)
    got = dart.quantize(x.cuda(), bits=bits, group_size=group, metadata_dtype=dtype, axis=-2)
    rows = x.transpose(1, 2)
    padded = torch.cat([rows, rows[..., -1:].expand(-1, -1, -tokens % group)], -1).contiguous()
    codes, scale, zero = expected(padded, bits, group)
    packed = pack(codes, bits)
    assert np.array_equal(to_np(got.values).reshape(packed.shape), packed)
    assert same(got.scale.reshape(scale.shape), scale) and same(got.zero_point.reshape(zero.shape), zero)


@pytest.mark.parametrize("rows", [1, 5, 37, 75, 150, 300])
@pytest.mark.parametrize("tokens", [1, 64, 127, 128, 129, 512, 1000, 4100])
def test_selection(rows, tokens):
    x = torch.randn(rows, 1, tokens, 128, generator=torch.Generator().manual_seed(rows + tokens)).half()
    got = dart.quantize_key_mixed(x.cuda(), group_size=32, promote_ratio=0.25, metadata_dtype=torch.float16).channel_indices.cpu()
    # fp16 sums are exact in double; the score is rounded to fp32, divided and rounded to fp16
    score = (x[:, 0].double().abs().sum(1).float() / torch.tensor(float(tokens))).half()
    order = torch.sort(score, dim=-1, descending=True, stable=True).indices[:, :32]
    assert torch.equal(got.reshape(rows, 32).long(), order)
