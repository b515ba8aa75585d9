"""C++ exceptions inside the native host path reach the caller as Python exceptions."""

import ctypes

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from dartkv_b200 import _lib


def test_a_tensor_without_storage_raises_instead_of_ending_the_process():
    # a fake CUDA tensor looks like a CUDA tensor until its storage (or the device) is asked for
    with FakeTensorMode(allow_non_fake_inputs=True):
        data = torch.empty(1, 1, 32, 32, device="cuda", dtype=torch.float16)
        desc = _lib.CacheDesc()
        desc.batch = desc.kv_heads = 1
        desc.head_dim = 32
        desc.dtype = _lib.F16
        address = ctypes.addressof(desc)
        with pytest.raises(RuntimeError):
            _lib.HOST.quantize(data, 2, 32, 3, _lib.F16, 0, 0)
        with pytest.raises(RuntimeError):
            _lib.HOST.quantize_mixed(data, 32, 8, _lib.F16, None, 0)
        with pytest.raises(RuntimeError):
            _lib.HOST.append(data, data, address, address, address, address, 0)
        with pytest.raises(RuntimeError):
            _lib.HOST.decode(data[:, :, 0], address, 0, 0, 1, 32, 1.0, 0, None)


def test_selection_without_a_score_buffer_is_refused_where_it_needs_one():
    # pointers are never dereferenced: nothing is launched
    def promote(dtype, head_dim, keys=0x10000000, count=8):
        return _lib.LIB.dartkv_promote_channels(keys, dtype, 2, 16, head_dim, 16 * head_dim, head_dim, count, None, 0x20000000, None)

    launches = _lib.LIB.dartkv_launch_count()
    for args in ((_lib.F32, 128), (_lib.BF16, 130), (_lib.F16, 63), (_lib.BF16, 128, 0x10000002)):
        assert promote(*args) == _lib.ELIMIT and "score buffer" in _lib.last_error()
    assert promote(_lib.F32, 128, count=0) == _lib.OK
    assert _lib.LIB.dartkv_launch_count() == launches
