"""The decoders' row between the host and the device (gpu.HostRow), over a library that copies host memory."""

from __future__ import annotations

import ctypes as C
from types import SimpleNamespace

import numpy as np
import pytest

from drama_rs_b200 import gpu


class FakeLib:
    def __init__(self) -> None:
        self.calls, self.held = [], []

    def dr_host_alloc(self, p, n):
        self.held.append(C.create_string_buffer(n))
        p._obj.value = C.addressof(self.held[-1])
        return 0

    def dr_h2d(self, d, h, n, st):
        self.calls.append("h2d")
        C.memmove(d, h, n)
        return 0

    def dr_d2h(self, h, d, n, st):
        self.calls.append("d2h")
        C.memmove(h, d, n)
        return 0

    def dr_host_free(self, p):
        return 0


@pytest.fixture
def row(monkeypatch):
    lib = FakeLib()
    monkeypatch.setattr(gpu.ffi, "lib", lambda: lib)
    dev = np.zeros(8, dtype=np.float32)
    r = gpu.HostRow(8, SimpleNamespace(raw=None, sync=lambda: lib.calls.append("sync")))
    return r, SimpleNamespace(ptr=dev.ctypes.data, nbytes=dev.nbytes), dev, lib.calls


@pytest.mark.parametrize("x", [np.arange(8.0), np.arange(8, dtype=np.float16), np.arange(8, dtype=np.int64), np.arange(16, dtype=np.float32)[::2],
                               np.arange(8, dtype=">f4").reshape(1, 8), np.array([0, 1, 2.5, 3, 4, 5, 6, 7], dtype=object)], ids=lambda a: str(a.dtype))
def test_rows_of_any_type_arrive_as_float32(row, x):
    r, buf, dev, _ = row
    r.put(buf, x)
    assert np.array_equal(dev, x.astype(np.float32).reshape(-1))
    assert np.array_equal(r.get(buf), dev)


def test_a_row_that_is_still_under_way_is_waited_for(row):
    r, buf, dev, calls = row
    r.put(buf, np.ones(8))
    r.put(buf, np.full(8, 2.0))
    first = r.get(buf)
    r.put(buf, np.zeros(3))
    assert calls == ["h2d", "sync", "h2d", "d2h", "sync", "h2d"]
    assert (first == 2).all() and np.array_equal(dev, [0, 0, 0, 2, 2, 2, 2, 2])
    with pytest.raises(AssertionError):
        r.put(buf, np.zeros(9))
