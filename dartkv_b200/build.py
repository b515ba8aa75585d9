"""Compile the native code of this package: the CUDA sources into ``libdartkv_b200.so`` (sm_100a only) and the
per-call host path into the CPython extension ``_dartkv_host.so``, which links against it.

``python dartkv_b200/build.py [--force] [-v]``; ``-v`` prints ptxas resource usage.  Extra nvcc flags can be
passed in ``DARTKV_NVCC_FLAGS``.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

PACKAGE_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PACKAGE_DIR, "csrc")
LIB_PATH = os.path.join(PACKAGE_DIR, "libdartkv_b200.so")
HOST_SOURCE = os.path.join(CSRC, "host_path.cpp")
HOST_PATH = os.path.join(PACKAGE_DIR, "_dartkv_host.so")
HOST_STAMP = os.path.join(PACKAGE_DIR, "build", "host_path.stamp")   # what the extension was built against
SOURCES = ("quantize.cu", "quantize_fast.cu", "cache_append.cu", "append_fast.cu", "materialize.cu", "decode_attention.cu", "decode_fast.cu", "decode_fused32.cu",
           "decode_wide.cu", "decode_rows.cu", "decode_many.cu", "decode_many_bf16.cu", "decode_many_bf16_f16.cu", "decode_many_f16_bf16.cu",
           "decode_many_f16.cu")
NVCC_FLAGS = (
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-O2",
)


def _nvcc() -> str:
    for candidate in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if candidate and os.path.exists(candidate):
            return candidate
    raise RuntimeError("nvcc not found; the dartkv_b200 kernels need the CUDA toolkit to build")


def _stale(sources) -> bool:
    if not os.path.exists(LIB_PATH):
        return True
    built = os.path.getmtime(LIB_PATH)
    headers = [os.path.join(CSRC, name) for name in os.listdir(CSRC) if name.endswith(".cuh")]
    deps = list(sources) + headers + [os.path.join(PACKAGE_DIR, "..", "include", "dartkv_b200.h")]
    return any(os.path.exists(p) and os.path.getmtime(p) > built for p in deps)


def _host_abi() -> str:
    """The C++ side of the installed torch and Python: an extension built against another one must not be loaded."""

    import torch

    return f"torch {torch.__version__} cxx11 {int(torch._C._GLIBCXX_USE_CXX11_ABI)} python {sys.version_info[:2]}"


def _host_stale() -> bool:
    if not (os.path.exists(HOST_PATH) and os.path.exists(HOST_STAMP)):
        return True
    header = os.path.join(PACKAGE_DIR, "..", "include", "dartkv_b200.h")
    if any(os.path.getmtime(p) > os.path.getmtime(HOST_PATH) for p in (HOST_SOURCE, header)):
        return True
    with open(HOST_STAMP) as stamp:
        return stamp.read() != _host_abi()


def _start_host_build(force: bool):
    """Start compiling the CPython extension (``None`` when it is up to date)."""

    if not force and not _host_stale():
        return None
    import torch
    from torch.utils import cpp_extension

    includes = [*cpp_extension.include_paths("cuda"), sysconfig.get_paths()["include"]]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-c", HOST_SOURCE, "-o", os.path.join(PACKAGE_DIR, "build", "host_path.o"),
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *[f"-I{path}" for path in includes]]
    return subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)


def _finish_host_build(proc) -> None:
    """Link the extension against the library beside it and torch's own libraries."""

    from torch.utils import cpp_extension

    out, _ = proc.communicate()
    if proc.returncode:
        print(out, file=sys.stderr)
        raise RuntimeError("g++ failed; see the compiler output above")
    libraries = [f"-L{path}" for path in cpp_extension.library_paths("cuda")]
    subprocess.run(["g++", "-shared", "-o", HOST_PATH, os.path.join(PACKAGE_DIR, "build", "host_path.o"), f"-L{PACKAGE_DIR}",
                    "-ldartkv_b200", "-Wl,-rpath,$ORIGIN", *libraries, "-ltorch_python", "-ltorch", "-ltorch_cpu",
                    "-lc10", "-lc10_cuda", "-lcudart"], check=True)
    with open(HOST_STAMP, "w") as stamp:
        stamp.write(_host_abi())


def build(force: bool = False, verbose: bool = False) -> str:
    """Build both shared objects in-tree and return the library's path (no-op when up to date)."""

    os.makedirs(os.path.join(PACKAGE_DIR, "build"), exist_ok=True)
    host = _start_host_build(force)
    path = _build_library(force, verbose)
    if host is not None:
        _finish_host_build(host)
    return path


def _build_library(force: bool, verbose: bool) -> str:

    sources = [os.path.join(CSRC, name) for name in SOURCES if os.path.exists(os.path.join(CSRC, name))]
    if not force and not _stale(sources):
        return LIB_PATH
    objects = []
    build_dir = os.path.join(PACKAGE_DIR, "build")
    procs = []
    for src in sources:
        obj = os.path.join(build_dir, os.path.basename(src) + ".o")
        objects.append(obj)
        cmd = [_nvcc(), *NVCC_FLAGS, *os.environ.get("DARTKV_NVCC_FLAGS", "").split(), "-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, proc in procs:
        out, _ = proc.communicate()
        if out.strip() and (verbose or proc.returncode):
            print(out, file=sys.stderr)
        failed |= proc.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed; see the compiler output above")
    link = [_nvcc(), "-shared", "-o", LIB_PATH, *objects, "-lcudart"]
    subprocess.run(link, check=True)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
