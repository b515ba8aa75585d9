"""Promoted channels are ranked by (score descending, channel ascending) whatever the keys hold: ties at the cut, all-zero
pages, infinities, and NaN as the largest score.  Every rank has one channel, so no slot of a page is left unwritten."""

import numpy as np
import pytest
import torch

import dartkv_b200 as dart

pytestmark = pytest.mark.gpu


def expected_ranks(keys):
    """[..., T, D] -> channels in rank order, from the score's bit pattern (exact sum, divided and rounded to the dtype)."""

    scores = (keys.double().abs().sum(-2).float() / keys.shape[-2]).to(keys.dtype)
    return order(scores)


def order(scores):
    bits = scores.view(torch.int32 if scores.dtype == torch.float32 else torch.int16).numpy().astype(np.int64)
    bits[scores.isnan().numpy()] = 0x7FFFFFFF
    return np.argsort(-bits, axis=-1, kind="stable")


def special_keys(kind, dtype, pages):
    gen = torch.Generator().manual_seed(7)
    keys = torch.randn(2, 3, 128 * pages, 128, generator=gen).to(dtype)
    if kind == "ties":          # scores of every fourth channel equal: the cut falls inside a tie
        keys = (torch.randint(1, 3, (2, 3, 1, 128), generator=gen) * torch.ones(128 * pages, 1)).to(dtype)
    if kind == "zero":
        keys.zero_()
    if kind == "wide":          # magnitudes far apart: more bits than a double holds in bf16
        scale = torch.exp2(torch.randint(-14, 14, keys.shape, generator=gen).float() * (4 if dtype == torch.bfloat16 else 0.5))
        keys = (keys.float() * scale).to(dtype)
    if kind == "nan_channel":   # one NaN: its channel ranks first
        keys[:, :, 5::128, 77] = float("nan")
    if kind == "nan_row":       # every score NaN
        keys[:, 1, 64::128, :] = float("nan")
    if kind == "some_nan":
        keys[:, :, 3::128, 1::3] = float("nan")
    if kind == "inf":
        keys[:, :, 9::128, 2::5] = float("-inf")
        keys[:, :, 11::128, 4::25] = float("nan")
    return keys


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("ratio", [0.25, 0.01, 0.9])
@pytest.mark.parametrize("kind", ["ties", "zero", "wide", "nan_channel", "nan_row", "some_nan", "inf"])
def test_pages_rank_each_channel_once(kind, ratio, dtype):
    keys = special_keys(kind, dtype, 2)
    ranks = expected_ranks(keys.unflatten(2, (2, 128)))
    cache = dart.DartKVCache(dart.DartKVCacheConfig(bits=2, page_size=128, key_group_size=128, value_group_size=64, sink_tokens=0,
                                                    hold_partial_pages=True, promote_ratio=ratio, metadata_dtype=dtype))
    cache.append(keys.cuda(), torch.zeros_like(keys).cuda())
    indices = [k.channel_indices.cpu().numpy() for k, _ in cache.iter_segments() if not isinstance(k, torch.Tensor)]
    assert len(indices) == 2
    for page, got in enumerate(indices):
        assert np.array_equal(got, ranks[:, :, page, :got.shape[-1]])


@pytest.mark.parametrize("kind", ["ties", "nan_channel", "nan_row", "some_nan", "inf"])
def test_general_page_kernel_ranks_each_channel_once(kind):
    keys = special_keys(kind, torch.float32, 1)[..., :100].contiguous()
    cache = dart.DartKVCache(dart.DartKVCacheConfig(bits=2, page_size=128, key_group_size=128, value_group_size=50, sink_tokens=0,
                                                    hold_partial_pages=True, promote_ratio=0.25))
    cache.append(keys.cuda(), torch.zeros_like(keys).cuda())
    (key, _), = cache.iter_segments()
    assert np.array_equal(key.channel_indices.cpu().numpy(), expected_ranks(keys)[..., :key.channel_indices.shape[-1]])


@pytest.mark.parametrize("dtype,head_dim", [(torch.float32, 128), (torch.bfloat16, 128), (torch.bfloat16, 130), (torch.float16, 63)])
@pytest.mark.parametrize("kind", ["ties", "zero", "wide", "nan_channel", "nan_row", "some_nan", "inf"])
def test_functional_selection_ranks_each_channel_once(dtype, head_dim, kind):
    keys = special_keys(kind, dtype, 1)
    keys = torch.cat([keys, keys[..., :2]], -1)[..., :head_dim].contiguous()
    ranks = expected_ranks(keys)
    mask, indices = dart.select_key_channels(keys.cuda(), 0.25)
    assert np.array_equal(indices.cpu().numpy(), ranks[..., :indices.shape[-1]])
    assert np.array_equal(mask.sum(-1).cpu().numpy(), np.full((2, 3), indices.shape[-1]))
    mixed = dart.quantize_key_mixed(keys.cuda(), group_size=128, promote_ratio=0.25, check_finite=False)
    assert torch.equal(mixed.channel_indices.long(), indices)
    # variance scores of such keys are NaN for whole rows: any order, but every channel once
    _, indices = dart.select_key_channels(keys.cuda(), 0.25, strategy="variance")
    assert indices.min() >= 0 and indices.max() < head_dim
    assert all(len(set(row.tolist())) == len(row) for row in indices.flatten(0, 1).cpu())
