"""The decode work split is host arithmetic: check, without a GPU, that every plan keeps a row's partials inside
the slots the workspace reserves for it, that the blocks' shares tile the units exactly, and that the workspace
bound covers every plan."""

import ctypes
import itertools

import pytest

from dartkv_b200 import _lib
from dartkv_b200._lib import LIB, CacheDesc, DecodePlanInfo, check


def make_desc(batch, heads, *, promoted=32, value_group=64, key_bits=2, value_bits=2, sink=32, dtype=_lib.BF16):
    d = CacheDesc()
    d.batch, d.kv_heads, d.head_dim = batch, heads, 128
    d.dtype = d.md_dtype = dtype
    d.page_size, d.key_group, d.value_group = 128, 128, value_group
    d.key_bits, d.value_bits = key_bits, value_bits
    d.key_mode = _lib.MIXED_PAGE if promoted else _lib.QUANTIZED_PAGE
    d.promoted = promoted
    d.sink_tokens, d.ring_tokens, d.regular_pages = sink, 128, 1
    d.max_key_pages, d.max_value_tokens = 4096, 4096 * 128
    check(LIB.dartkv_cache_geometry(ctypes.byref(d)))
    for i, name in enumerate(("k_sink", "v_sink", "k_ring", "v_ring", "k_pages", "v_codes", "v_meta", "page_start",
                              "page_tokens", "state")):
        setattr(d, name, 0x10000000 + 0x1000000 * i)   # never dereferenced: only their alignment is looked at
    return d


def block_of_unit(x, blocks, units):
    j = x * blocks // units
    if (j + 1) * units // blocks <= x:
        j += 1
    return j


def plan(d, q_dtype, hq, flavour, tokens):
    info = DecodePlanInfo()
    check(LIB.dartkv_decode_plan(ctypes.byref(d), q_dtype, hq, flavour, tokens, ctypes.byref(info)))
    return info


def pages_of_blocks(info, row, pages):
    """The pages of a work row that each block works on, as the kernels find them."""
    parts = []
    for j in range(info.stream_blocks):
        begin, end = j * info.units // info.stream_blocks, (j + 1) * info.units // info.stream_blocks
        begin, end = max(begin - row * info.quads, 0), min(end - row * info.quads, info.quads)
        if begin < end:
            parts.append(range(info.unit_pages * begin, min(info.unit_pages * end, pages)))
    return parts


ROWS = [(1, 1), (1, 8), (2, 8), (3, 2), (5, 2), (10, 2), (6, 8), (16, 8), (32, 8), (37, 8), (128, 8), (512, 8)]
TOKENS = [1, 31, 32, 33, 159, 160, 161, 32 + 4 * 128, 32 + 5 * 128 + 77, 8192, 32 + 116 * 128, 32 + 225 * 128, 32 + 228 * 128, 32768,
          32 + 289 * 128, 131072]


@pytest.mark.parametrize("split", [None, "aligned", "unaligned", "unaligned:7", "unaligned:3"])
@pytest.mark.parametrize("flavour", [_lib.DEQUANT_PER_OP, _lib.DEQUANT_FUSED])
def test_tensor_core_plans_stay_inside_their_partial_slots(flavour, split, decode_split):
    decode_split(split)
    for (batch, heads), tokens in itertools.product(ROWS, TOKENS):
        d = make_desc(batch, heads)
        info = plan(d, _lib.BF16, 4 * heads, flavour, tokens)
        assert info.kernel == (1 if flavour == _lib.DEQUANT_PER_OP else 2)
        rows = batch * heads
        pages = max(1, (tokens - 32) // 128)
        assert info.unit_pages in (4, 8) and info.row_groups == 1
        assert info.quads == -(-pages // info.unit_pages)
        assert info.units == rows * info.quads
        assert 1 <= info.stream_blocks <= info.units
        assert 2 <= info.total_splits <= 17
        # the shares tile the units
        edges = [j * info.units // info.stream_blocks for j in range(info.stream_blocks + 1)]
        assert edges[0] == 0 and edges[-1] == info.units and all(a < b for a, b in zip(edges, edges[1:]))
        # every row's dense slot + stream blocks fit its slots (first, middle and last rows are representative;
        # small cases check every row)
        sample = range(rows) if rows <= 64 else (0, 1, rows // 3, rows // 2, rows - 2, rows - 1)
        for row in sample:
            first = block_of_unit(row * info.quads, info.stream_blocks, info.units)
            last = block_of_unit(row * info.quads + info.quads - 1, info.stream_blocks, info.units)
            assert edges[first] <= row * info.quads < edges[first + 1]
            assert 1 + (last - first + 1) <= info.total_splits
        if rows <= 64:
            for row in range(rows):
                parts = pages_of_blocks(info, row, pages)
                assert [p for part in parts for p in part] == list(range(pages)) and 1 + len(parts) <= info.total_splits
        need = 16 + batch * 4 * heads * info.total_splits * (2 + 128) * 4
        assert LIB.dartkv_decode_workspace_bytes(ctypes.byref(d), 4 * heads, tokens) >= need


@pytest.mark.parametrize("flavour", [_lib.DEQUANT_PER_OP, _lib.DEQUANT_FUSED])
def test_slots_are_those_of_the_units_that_are_dealt_out(flavour):
    # units of eight pages whose shares end inside a row: counted in units of four, 5 x 2 rows of 225 to 228 pages took 21 slots, more
    # than the merge of tensor-core layouts is made for, and 6 x 8 of 289 to 296 nine, one more than the warp-per-row merge takes
    for (batch, heads), pages, most in (((5, 2), range(225, 229), 17), ((10, 2), range(225, 229), 17), ((6, 8), range(289, 297), 8)):
        for n in pages:
            info = plan(make_desc(batch, heads), _lib.BF16, 4 * heads, flavour, 32 + 128 * n)
            assert info.total_splits <= most
            assert all(1 + len(pages_of_blocks(info, row, n)) <= info.total_splits for row in range(batch * heads))


def test_other_geometries_take_the_general_tensor_core_kernel():
    for kwargs in (dict(value_bits=4), dict(key_bits=4, promoted=0), dict(value_group=32), dict(value_bits=8, key_bits=8, promoted=0)):
        d = make_desc(2, 2, **kwargs)
        for flavour in (_lib.DEQUANT_PER_OP, _lib.DEQUANT_FP32):
            info = plan(d, _lib.BF16, 8, flavour, 5000)
            assert info.kernel == 3 and info.stream_blocks >= 1 and info.generic_splits == 0
            assert info.quads == (max(1, (5000 - 32) // 128) + 3) // 4 and 2 <= info.total_splits <= 17
        # the unrounded flavour of these geometries has no 16-bit tile to go through: CUDA-core kernel
        info = plan(d, _lib.BF16, 8, _lib.DEQUANT_FUSED, 5000)
        assert info.kernel == 0 and info.stream_blocks == 0 and info.generic_splits >= 1
        assert info.total_splits == info.generic_splits
    d = make_desc(2, 2)
    assert plan(d, _lib.F32, 8, _lib.DEQUANT_PER_OP, 5000).kernel == 0      # query dtype differs from the cache dtype
    assert plan(d, _lib.BF16, 8, _lib.DEQUANT_FP32, 5000).kernel == 3       # the fp32 flavour of the headline geometry
    assert plan(d, _lib.BF16, 16, _lib.DEQUANT_PER_OP, 5000).kernel == 0    # 8 query heads per kv head
    d.md_dtype = _lib.F16                                                    # fp16 metadata beside a bf16 cache
    assert plan(d, _lib.BF16, 8, _lib.DEQUANT_PER_OP, 5000).kernel == 1     # the per-op kernel casts its operands
    assert plan(d, _lib.BF16, 8, _lib.DEQUANT_FP32, 5000).kernel == 3
    assert plan(d, _lib.BF16, 8, _lib.DEQUANT_FUSED, 5000).kernel == 2


def test_plan_argument_errors():
    d = make_desc(1, 2)
    info = DecodePlanInfo()
    assert LIB.dartkv_decode_plan(ctypes.byref(d), _lib.BF16, 3, 0, 100, ctypes.byref(info)) == -1
    assert LIB.dartkv_decode_plan(ctypes.byref(d), _lib.BF16, 8, 9, 100, ctypes.byref(info)) == -1
    assert LIB.dartkv_decode_plan(ctypes.byref(d), _lib.BF16, 8, 0, 0, ctypes.byref(info)) == -1


@pytest.mark.parametrize("kwargs", [dict(value_bits=4), dict(key_bits=4, promoted=0), dict(value_group=32), dict()],
                         ids=["v4", "k4", "vg32", "headline"])
def test_workspace_bound_covers_every_smaller_token_count(kwargs):
    # a workspace sized for a capacity must serve every token count up to it, for every query dtype and flavour
    # (the generic split count is not monotonic in the token count: its chunk is rounded up to whole tiles)
    for batch, heads, hq in ((2, 8, 32), (1, 8, 32), (1, 1, 4), (16, 8, 32)):
        d = make_desc(batch, heads, **kwargs)
        for capacity in (300, 3000, 4256, 8352):
            have = LIB.dartkv_decode_workspace_bytes(ctypes.byref(d), hq, capacity)
            worst = 0
            for tokens in range(1, capacity + 1, 1 if capacity <= 3000 else 7):
                for q_dtype, flavour in ((_lib.BF16, _lib.DEQUANT_PER_OP), (_lib.F32, _lib.DEQUANT_PER_OP),
                                         (_lib.BF16, _lib.DEQUANT_FUSED)):
                    info = plan(d, q_dtype, hq, flavour, tokens)
                    worst = max(worst, 16 + batch * hq * info.total_splits * (2 + 128) * 4)
            assert have >= worst, (kwargs, batch, heads, capacity, have, worst)


@pytest.mark.parametrize("kwargs,flavour", [(dict(), _lib.DEQUANT_PER_OP), (dict(), _lib.DEQUANT_FUSED), (dict(), _lib.DEQUANT_FP32),
                                            (dict(value_bits=4, key_bits=4, promoted=0), _lib.DEQUANT_PER_OP)])
def test_a_query_from_an_odd_element_on_is_refused_before_any_launch(kwargs, flavour):
    d = make_desc(1, 2, **kwargs)
    query, workspace, out = 0x20000002, 0x30000000, 0x40000000       # never dereferenced
    for call, rep in ((LIB.dartkv_decode_attention, 4), (LIB.dartkv_decode_attention_padded, 4), (LIB.dartkv_decode_attention_rows, 8)):
        if rep > 4 and flavour != _lib.DEQUANT_PER_OP:
            continue
        padding = [] if call is LIB.dartkv_decode_attention else [None]
        args = [ctypes.byref(d), query, _lib.BF16, 2 * rep, 0.1, flavour, 5000, *padding, workspace, 1 << 40, out, None]
        assert call(*args) == _lib.EINVAL and "aligned" in _lib.last_error()


@pytest.mark.parametrize("query_heads,dtype", [(4, _lib.BF16), (4, _lib.F32)])
def test_a_workspace_from_an_odd_byte_on_is_refused_before_any_launch(query_heads, dtype):
    d = make_desc(1, 1, dtype=dtype)
    for offset in (1, 2, 3, 6):
        assert LIB.dartkv_decode_attention(ctypes.byref(d), 0x20000000, dtype, query_heads, 0.1, _lib.DEQUANT_PER_OP, 5000,
                                           0x30000000 + offset, 1 << 40, 0x40000000, None) == _lib.EINVAL
        assert "workspace" in _lib.last_error()


def test_the_scratch_of_a_class_of_widths_serves_every_width_in_it():
    # calls of 5..8, 9..16, ... query heads per KV head share the buffer of the widest
    for kwargs in (dict(), dict(value_bits=4, key_bits=4, promoted=0), dict(value_group=32), dict(dtype=_lib.F32)):
        for (batch, heads), capacity in itertools.product([(1, 1), (2, 8), (128, 8)], [300, 3000, 40000]):
            d = make_desc(batch, heads, **kwargs)
            for low, high in ((5, 8), (9, 16), (17, 32), (33, 64)):
                most = LIB.dartkv_decode_workspace_bytes(ctypes.byref(d), high * heads, capacity)
                assert all(LIB.dartkv_decode_workspace_bytes(ctypes.byref(d), rep * heads, capacity) <= most
                           for rep in range(low, high))


def test_cuda_core_plans_give_every_sm_blocks_where_there_are_tiles():
    for (batch, heads), tokens in itertools.product([(1, 1), (1, 2), (1, 8), (4, 8), (37, 8)], [31, 1000, 32768, 131072]):
        info = plan(make_desc(batch, heads, dtype=_lib.F32), _lib.F32, 4 * heads, _lib.DEQUANT_PER_OP, tokens)
        rows, tiles = batch * heads, -(-tokens // 32)
        assert info.kernel == 0 and info.total_splits == info.generic_splits <= tiles
        # rounding a split up to whole tiles costs at most half of the blocks
        assert rows * info.generic_splits >= min(rows * tiles, 2 * 148)


@pytest.mark.parametrize("split", [None, "aligned", "unaligned", "unaligned:7"])
def test_many_row_plans_stay_inside_their_partial_slots(split, decode_split):
    decode_split(split)
    info = DecodePlanInfo()
    for (batch, heads), tokens in itertools.product([(1, 1), (2, 8), (37, 8), (128, 8)], [1024, 1183, 8192, 32768 + 77, 131072]):
        d = make_desc(batch, heads)
        for rep in (5, 7, 8, 9, 16, 17, 20, 31, 33, 49, 57, 64):
            assert plan(d, _lib.BF16, rep * heads, _lib.DEQUANT_PER_OP, tokens).kernel == 0      # the ordinary entry point
            check(LIB.dartkv_decode_plan_rows(ctypes.byref(d), _lib.BF16, rep * heads, _lib.DEQUANT_PER_OP, tokens, ctypes.byref(info)))
            # groups of eight query rows, or of 32 where a block restores a page once for all rows of a group
            assert info.row_groups == (-(-rep // 8) if info.unit_pages else -(-rep // 32))
            assert info.unit_pages == 4 or (info.unit_pages == 0 and rep > 8)
            rows = batch * heads * info.row_groups
            assert info.kernel == 4 and info.quads == ((tokens - 32) // 128 + 3) // 4 and info.units == rows * info.quads
            assert 1 <= info.stream_blocks <= info.units and 2 <= info.total_splits <= 17
            sample = range(rows) if rows <= 64 else (0, 1, rows // 3, rows // 2, rows - 2, rows - 1)
            for row in sample:
                first = block_of_unit(row * info.quads, info.stream_blocks, info.units)
                last = block_of_unit(row * info.quads + info.quads - 1, info.stream_blocks, info.units)
                assert 1 + (last - first + 1) <= info.total_splits
                if info.unit_pages == 0:   # blocks of one work row each, as many for every row
                    assert (first, last) == (row * (info.stream_blocks // rows), (row + 1) * (info.stream_blocks // rows) - 1)
            assert info.unit_pages == 4 or info.stream_blocks % rows == 0 and info.total_splits == 1 + info.stream_blocks // rows
            need = 16 + batch * rep * heads * info.total_splits * (2 + 128) * 4
            assert LIB.dartkv_decode_workspace_bytes(ctypes.byref(d), rep * heads, tokens) >= need
        # up to four rows, and what the many-row kernel does not take, run as through the ordinary entry point
        for hq, flavour in ((4 * heads, _lib.DEQUANT_PER_OP), (4 * heads, _lib.DEQUANT_FUSED), (8 * heads, _lib.DEQUANT_FUSED),
                            (8 * heads, _lib.DEQUANT_FP32), (65 * heads, _lib.DEQUANT_PER_OP)):
            check(LIB.dartkv_decode_plan_rows(ctypes.byref(d), _lib.BF16, hq, flavour, tokens, ctypes.byref(info)))
            ordinary = plan(d, _lib.BF16, hq, flavour, tokens)
            assert bytes(info) == bytes(ordinary)


@pytest.mark.parametrize("pool", ["k_sink", "v_sink", "k_ring", "v_ring"])
def test_dense_pools_that_sixteen_byte_loads_cannot_read_stay_with_the_narrower_kernel(pool):
    d, info = make_desc(8, 8), DecodePlanInfo()
    for offset, unit_pages in ((0, 0), (8, 4), (16, 0)):
        setattr(d, pool, 0x70000000 + offset)
        check(LIB.dartkv_decode_plan_rows(ctypes.byref(d), _lib.BF16, 20 * 8, _lib.DEQUANT_PER_OP, 4096, ctypes.byref(info)))
        assert info.kernel == 4 and info.unit_pages == unit_pages


@pytest.mark.parametrize("batch,rep,tokens,once_for_all", [(1, 64, 1100, False), (1, 48, 2100, False), (2, 48, 1100, True), (1, 64, 2100, True),
                                                           (8, 20, 4096, True), (1, 20, 4096, False), (8, 9, 1100, True)])
def test_pages_are_restored_once_for_all_rows_where_that_is_faster(batch, rep, tokens, once_for_all):
    info = DecodePlanInfo()
    check(LIB.dartkv_decode_plan_rows(ctypes.byref(make_desc(batch, 8)), _lib.BF16, 8 * rep, _lib.DEQUANT_PER_OP, tokens, ctypes.byref(info)))
    assert (info.unit_pages == 0) == once_for_all
