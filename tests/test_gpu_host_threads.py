"""A native call whose launch waits for room in the GPU's queue leaves the other Python threads running, whatever they do meanwhile."""

import gc
import threading
import time
import types
import weakref

import pytest
import torch

import dartkv_b200 as dart

pytestmark = pytest.mark.gpu


def calls():
    data = torch.randn(1, 2, 200, 128, device="cuda", dtype=torch.float16)
    config = dart.DartKVCacheConfig(bits=2, page_size=128, key_group_size=128, value_group_size=64, sink_tokens=4, hold_partial_pages=True)
    cache = dart.DartKVCache(config)
    cache.append(data, data)
    packed, mixed = dart.quantize(data), dart.quantize_key_mixed(data)

    def new_cache():
        dart.DartKVCache(config, max_tokens=300).append(data, data)

    return {"get": cache.get, "dequantize": packed.dequantize, "dequantize_mixed": mixed.dequantize, "new_cache": new_cache,
            "quantize": lambda: dart.quantize(data, check_finite=False), "quantize_mixed": lambda: dart.quantize_key_mixed(data, check_finite=False)}


@pytest.mark.parametrize("name", ["get", "dequantize", "dequantize_mixed", "new_cache", "quantize", "quantize_mixed"])
def test_other_threads_run_while_a_launch_waits(name):
    call = calls()[name]
    call()
    torch.cuda.synchronize()
    done, error = threading.Event(), []

    def work():
        try:
            torch.cuda._sleep(int(0.8 * 1.9e9))    # some 0.8 s of a GPU that spins
            for _ in range(2500):                  # more launches than the queue has room for
                call()
        except Exception as e:
            error.append(e)
        done.set()

    thread = threading.Thread(target=work)
    start = last = time.perf_counter()
    longest = 0.0
    thread.start()
    while not done.is_set():
        time.sleep(0.001)
        now = time.perf_counter()
        longest, last = max(longest, now - last), now
    thread.join()
    torch.cuda.synchronize()
    assert not error, error
    assert last - start > 0.4                      # the thread did wait for the GPU
    assert longest < 0.2, longest                  # and this one did not


def test_the_descriptor_outlives_a_call_that_reads_it(monkeypatch):
    cache = calls()["get"].__self__
    desc, seen = weakref.ref(cache._desc), []

    def get(*args):
        cache.clear()                              # what another thread may do while the interpreter is unlocked
        gc.collect()
        seen.append(desc() is not None)
        return ()

    monkeypatch.setattr(dart._lib, "HOST", types.SimpleNamespace(get=get))
    cache.get()
    assert seen == [True]
