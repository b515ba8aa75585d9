"""Groups with Inf or NaN (``check_finite=False``), and groups of finite elements whose range overflows: the kernels for whole
code words give the bytes of the element-by-element arithmetic, clamp(rint((x - min) / scale), 0, qmax) with minimum and
maximum over the elements that are not NaN and code 0 for a NaN quotient."""

import numpy as np
import pytest
import torch

import dartkv_b200 as dart
from tests.helpers import to_np

pytestmark = pytest.mark.gpu


def expected(x, bits, group, qmax=None):
    """x [rows, n] (n a multiple of group) -> codes, scale, zero point by the rules above, every step rounded to x's dtype."""

    x = x.cpu().unflatten(-1, (-1, group))
    nan = x.isnan()
    mn = x.masked_fill(nan, float("inf")).amin(-1, keepdim=True)
    mx = x.masked_fill(nan, float("-inf")).amax(-1, keepdim=True)
    qmax = float(2 ** bits - 1) if qmax is None else qmax
    spread = mx - mn
    eps = torch.tensor(1e-4).to(x.dtype)
    spread = torch.where(spread > eps, spread, eps)      # a NaN range (all Inf) becomes the smallest one too
    scale = (spread.float() / qmax).to(x.dtype)
    ratio = ((x - mn).float() / scale.float()).to(x.dtype)
    codes = torch.minimum(ratio.float().round().nan_to_num(0.0, float("inf"), 0.0).clamp_min(0), torch.as_tensor(qmax)).to(torch.uint8)
    return codes.flatten(-2), scale[..., 0], mn[..., 0]


def pack(codes, bits):
    v = to_np(codes).astype(np.int64).reshape(*codes.shape[:-1], -1, 8 // bits)
    return (v << (bits * np.arange(8 // bits))).sum(-1).astype(np.uint8)


def data(dtype, kind, *shape):
    gen = torch.Generator().manual_seed(11)
    x = torch.randn(*shape, generator=gen)
    if kind == "overflow":
        x = x.sign() * torch.finfo(dtype).max * (0.6 + 0.3 * torch.rand(*shape, generator=gen))
        return x.to(dtype)
    x = x.to(dtype)
    for value, share in {"nan": [(float("nan"), 50)], "inf": [(float("inf"), 90), (float("-inf"), 110)],
                         "both": [(float("nan"), 70), (float("inf"), 130)], "all_nan": [(float("nan"), 1)]}[kind]:
        x[torch.rand(*shape, generator=gen) < 1 / share] = value
    return x


def same(got, ref):
    return np.array_equal(to_np(got), to_np(ref), equal_nan=True)


KINDS = ["nan", "inf", "both", "all_nan", "overflow"]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("bits,group,axis", [(2, 8, -1), (2, 64, -1), (4, 128, -1), (8, 256, -1), (2, 64, 1), (4, 32, 1), (8, 16, 1)])
def test_uniform(dtype, kind, bits, group, axis):
    x = data(dtype, kind, 3, 256, 256)
    q = dart.quantize(x.cuda(), bits=bits, group_size=group, axis=axis, check_finite=False)
    codes, scale, zero = expected(x.movedim(axis, -1).contiguous(), bits, group)
    assert same(q.scale, scale) and same(q.zero_point, zero)
    assert np.array_equal(to_np(q.values), pack(codes, bits))
    if kind != "overflow":
        with pytest.raises(ValueError, match="finite"):
            dart.quantize(x.cuda(), bits=bits, group_size=group, axis=axis)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kind", KINDS)
def test_mixed_keys(dtype, kind):
    x = data(dtype, kind, 2, 2, 256, 96)
    indices = torch.arange(1, 96, 4).expand(2, 2, -1)
    q = dart.quantize_key_mixed(x.cuda(), group_size=64, indices=indices.cuda(), check_finite=False)
    qmax = torch.full((96, 1, 1), 3.0)
    qmax[1::4] = 15.0
    codes, scale, zero = expected(x.transpose(2, 3).contiguous(), 2, 64, qmax)
    assert same(q.scale, scale) and same(q.zero_point, zero)
    codes = codes.unflatten(-1, (-1, 64))
    assert np.array_equal(to_np(q.low_values), pack(codes & 3, 2))
    assert np.array_equal(to_np(q.high_values), pack(codes[:, :, 1::4] >> 2, 2))
    if kind != "overflow":
        with pytest.raises(ValueError, match="finite"):
            dart.quantize_key_mixed(x.cuda(), group_size=64, indices=indices.cuda())
