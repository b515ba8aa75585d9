"""The build notices when the CPython extension no longer fits the installed torch or Python."""

import os
import time

from dartkv_b200 import build


def test_extension_is_rebuilt_for_another_torch_or_source(tmp_path, monkeypatch):
    built, stamp, source = tmp_path / "host.so", tmp_path / "host.stamp", tmp_path / "host_path.cpp"
    for name, path in (("HOST_PATH", built), ("HOST_STAMP", stamp), ("HOST_SOURCE", source)):
        monkeypatch.setattr(build, name, str(path))
    source.write_text("")
    assert build._host_stale()                       # never built
    built.write_text("")
    os.utime(built, (time.time() + 60, time.time() + 60))
    assert build._host_stale()                       # built by something that left no stamp
    stamp.write_text(build._host_abi())
    assert not build._host_stale()
    monkeypatch.setattr("torch.__version__", "0.0.0")
    assert build._host_stale()                       # torch was replaced
    monkeypatch.undo()
    for name, path in (("HOST_PATH", built), ("HOST_STAMP", stamp), ("HOST_SOURCE", source)):
        monkeypatch.setattr(build, name, str(path))
    assert not build._host_stale()
    os.utime(source, (time.time() + 120, time.time() + 120))
    assert build._host_stale()                       # the source is newer
