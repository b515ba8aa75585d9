"""A process's first call of a kernel loads that kernel and not every variant of it."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import time, torch, dartkv_b200 as dart
cache = dart.DartKVCache(dart.DartKVCacheConfig(bits=2, page_size=128, key_group_size=128, value_group_size=64, sink_tokens=32,
                                                hold_partial_pages=True, metadata_dtype=torch.bfloat16, promote_ratio=0.25))
data = torch.randn(8, 8, 4096, 128, device="cuda", dtype=torch.bfloat16)
cache.append(data, data)
for rows in (4, 8, 20):                     # the last one is the first that restores a page once for all rows
    query = torch.randn(8, 8 * rows, 1, 128, device="cuda", dtype=torch.bfloat16)
    cache.decode_workspace(8 * rows)
    torch.cuda.synchronize()
    start = time.perf_counter()
    dart.fused_dart_attention(query, cache, fallback=False)
    torch.cuda.synchronize()
    took = time.perf_counter() - start
print("TOOK", 1e3 * took)
"""


def test_first_call_of_many_rows():
    # 37 ms with all variants in one module, about 4 ms with those of a pair of types: the fastest of three processes counts
    took = []
    for _ in range(3):
        done = subprocess.run([sys.executable, "-c", CODE], capture_output=True, text=True, timeout=300,
                              cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
        assert done.returncode == 0, done.stderr[-2000:]
        took.append(float(done.stdout.split("TOOK")[1]))
        if took[-1] < 15:
            return
    assert min(took) < 15, took
