"""The arrays that a prefill step reads back and sends (gpu.PinnedPair), over a library that copies host memory."""

from __future__ import annotations

import ctypes as C
from types import SimpleNamespace

import numpy as np
import pytest

from drama_rs_b200 import gpu


@pytest.mark.parametrize("count", [1, 2, 256])
def test_offsets_of_counts(monkeypatch, count):
    calls, held = [], []

    def alloc(p, n):
        held.append(C.create_string_buffer(b"\xaa" * n, n))
        p._obj.value = C.addressof(held[-1])
        return 0

    def copy(name):
        return lambda d, s, n, st: calls.append(name) or C.memmove(d, s, n) and 0

    lib = SimpleNamespace(dr_host_alloc=alloc, dr_host_free=lambda p: calls.append("free") or 0, dr_d2h=copy("d2h"), dr_h2d=copy("h2d"))
    monkeypatch.setattr(gpu.ffi, "lib", lambda: lib)
    counts, offsets = np.arange(1, count + 1, dtype=np.int32), np.full(count, -1, dtype=np.int32)
    dev = lambda a: SimpleNamespace(ptr=a.ctypes.data)
    pair = gpu.PinnedPair(count, np.int32, SimpleNamespace(raw=None, sync=lambda: calls.append("sync")))
    for _ in range(2):
        got = pair.get(dev(counts))
        np.cumsum(got[:-1], out=pair.out[1:])
        pair.put(dev(offsets))
        assert np.array_equal(offsets, np.cumsum(counts) - counts)
        counts += 3
    assert calls == ["d2h", "sync", "h2d"] * 2
    del pair, got
    assert calls[-2:] == ["sync", "free"]
