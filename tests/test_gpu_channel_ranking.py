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
    bits = scores.view(torch.int16).numpy().astype(np.int64)
    bits[np.isnan(scores.float().numpy())] = 0x7FFF
    return np.argsort(-bits, axis=-1, kind="stable")


def special_keys(kind, dtype, pages):
    gen = torch.Generator().manual_seed(7)
    keys = torch.randn(2, 3, 128 * pages, 128, generator=gen).to(dtype)
    if kind == "ties":          # scores of every fourth channel equal: the cut falls inside a tie
        keys = (torch.randint(1, 3, (2, 3, 1, 128), generator=gen) * torch.ones(128 * pages, 1)).to(dtype)
    if kind == "zero":
        keys.zero_()
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
@pytest.mark.parametrize("kind", ["ties", "zero", "nan_channel", "nan_row", "some_nan", "inf"])
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
