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
