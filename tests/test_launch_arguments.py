"""The launch helper takes arguments that a kernel's parameters can be initialised with, and refuses others when it is compiled."""

import os
import subprocess

import pytest

from dartkv_b200 import build

SOURCE = """
#include "common.cuh"
__global__ void scale_kernel(float* data, const int32_t* index, int64_t n, float by) { if (index && n) data[0] *= by; }
cudaError_t launch(float* data, int32_t* index, int n) { return launch_following(scale_kernel, dim3(1), dim3(32), 0, nullptr, %s); }
"""


@pytest.mark.parametrize("arguments,compiles", [("data, index, n, 2.0f", True), ("data, index, n, 2.0", True), ("index, index, n, 2.0f", False),
                                                ("data, index, index, 2.0f", False), ("data, n, n, 2.0f", False)])
def test_arguments_are_checked(tmp_path, arguments, compiles):
    try:
        nvcc = build._nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    source = tmp_path / "launch.cu"
    source.write_text(SOURCE % arguments)
    done = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", build.CSRC, "-I", os.path.join(build.CSRC, "../../include"),
                           "-c", str(source), "-o", str(tmp_path / "launch.o")], capture_output=True, text=True, timeout=300)
    assert (done.returncode == 0) == compiles, done.stderr
    assert compiles or "static_cast" in done.stderr or "invalid type conversion" in done.stderr, done.stderr
