"""Thin RAII wrappers over device memory, streams and graphs through the C ABI.

The host-side mirror of the reference's src/gpu.rs: `check` (gpu.rs:9-15), `launched`
(gpu.rs:18-26), `DevBuf` (gpu.rs:35-120), `Stream` (gpu.rs:122-136), `Graph` (gpu.rs:138-163).
Everything goes through dr_* calls; torch is not involved.
"""

from __future__ import annotations

import ctypes as C

import numpy as np

from . import ffi


def check(code: int, what: str) -> None:
    if code != 0:
        msg = ffi.lib().dr_error_string(code).decode()
        raise RuntimeError(f"{what}: CUDA error {code} ({msg})")


def launched(code: int, what: str, debug: bool = True) -> None:
    """Status of a kernel launcher: its own argument check, then (debug) the launch error."""
    if code != 0:
        raise RuntimeError(f"{what}: unsupported shape (launcher returned {code})")
    if debug:
        check(ffi.lib().dr_last_error(), what)


class Stream:
    def __init__(self) -> None:
        self.raw = C.c_void_p()
        check(ffi.lib().dr_stream_create(C.byref(self.raw)), "stream_create")

    def sync(self) -> None:
        check(ffi.lib().dr_stream_sync(self.raw), "stream_sync")

    def close(self) -> None:
        if self.raw:
            ffi.lib().dr_stream_destroy(self.raw)
            self.raw = C.c_void_p()


class DevBuf:
    """A device allocation; pointers handed to kernels stay valid for its lifetime."""

    def __init__(self, nbytes: int) -> None:
        self.nbytes = int(nbytes)
        self._p = C.c_void_p()
        check(ffi.lib().dr_malloc(C.byref(self._p), max(self.nbytes, 16)), "malloc")

    @classmethod
    def from_array(cls, a: np.ndarray, st: Stream) -> "DevBuf":
        a = np.ascontiguousarray(a)
        b = cls(a.nbytes)
        if a.nbytes:
            check(ffi.lib().dr_h2d(b._p, a.ctypes.data_as(C.c_void_p), a.nbytes, st.raw), "h2d")
            st.sync()  # the host array may be a temporary
        return b

    @classmethod
    def zeros(cls, nbytes: int, st: Stream) -> "DevBuf":
        b = cls(nbytes)
        b.zero(st)
        return b

    @property
    def ptr(self) -> int:
        return self._p.value or 0

    def at(self, byte_offset: int) -> C.c_void_p:
        return C.c_void_p(self.ptr + int(byte_offset))

    def zero(self, st: Stream) -> None:
        check(ffi.lib().dr_memset(self._p, 0, self.nbytes, st.raw), "memset")

    def fill(self, byte: int, st: Stream) -> None:
        check(ffi.lib().dr_memset(self._p, byte, self.nbytes, st.raw), "memset")

    def upload(self, a: np.ndarray, st: Stream, byte_offset: int = 0) -> None:
        a = np.ascontiguousarray(a)
        assert byte_offset + a.nbytes <= self.nbytes
        check(ffi.lib().dr_h2d(self.at(byte_offset), a.ctypes.data_as(C.c_void_p), a.nbytes, st.raw), "h2d")
        st.sync()

    def download(self, dtype, count: int, st: Stream, byte_offset: int = 0) -> np.ndarray:
        out = np.empty(count, dtype=dtype)
        assert byte_offset + out.nbytes <= self.nbytes
        check(ffi.lib().dr_d2h(out.ctypes.data_as(C.c_void_p), self.at(byte_offset), out.nbytes, st.raw), "d2h")
        st.sync()
        return out

    def free(self) -> None:
        if self._p:
            ffi.lib().dr_free(self._p)
            self._p = C.c_void_p()

    def __del__(self) -> None:
        try:
            self.free()
        except Exception:
            pass


class Graph:
    """Capture `record()` (a callable that issues launches on `st`) once; replay with launch()."""

    def __init__(self, st: Stream, record) -> None:
        l = ffi.lib()
        check(l.dr_graph_begin(st.raw), "graph_begin")
        try:
            record()
        except Exception:
            tmp = C.c_void_p()
            l.dr_graph_end(st.raw, C.byref(tmp))
            raise
        self.exec = C.c_void_p()
        check(l.dr_graph_end(st.raw, C.byref(self.exec)), "graph_end")

    def launch(self, st: Stream) -> None:
        check(ffi.lib().dr_graph_launch(self.exec, st.raw), "graph_launch")

    def destroy(self) -> None:
        if self.exec:
            ffi.lib().dr_graph_destroy(self.exec)
            self.exec = C.c_void_p()


class HostRow:
    """A row of floats that crosses between the host and the front of a device buffer on every step. Both directions go
    through pinned memory of the row's own, so that the copies are queued behind one another and the host waits once, for the
    result (pageable memory made every step two staged copies with a wait each: 146 us a step of 112 us of kernels, 130 so).
    Copies by a kernel of one block, in a graph or beside it, and a word in pinned memory that the host watches instead of
    the stream measured the same or slower."""

    def __init__(self, count: int, st: Stream) -> None:
        self._l, self._st = ffi.lib(), st
        self._p = C.c_void_p()
        check(self._l.dr_host_alloc(C.byref(self._p), 8 * count), "host_alloc")
        both = np.frombuffer((C.c_float * (2 * count)).from_address(self._p.value), dtype=np.float32)
        self._in, self._out, self._out_p = both[:count], both[count:], C.c_void_p(self._p.value + 4 * count)
        self._queued = False  # a copy out of _in may still be under way

    def put(self, dev, x: np.ndarray) -> None:
        n = x.size
        assert n <= self._in.size and 4 * n <= dev.nbytes
        if self._queued:
            self._st.sync()
        np.copyto(self._in if n == self._in.size else self._in[:n], x.reshape(-1), casting="unsafe")  # as astype(np.float32) takes it
        self._queued = True
        check(self._l.dr_h2d(dev.ptr, self._p, 4 * n, self._st.raw), "h2d")

    def get(self, dev) -> np.ndarray:
        check(self._l.dr_d2h(self._out_p, dev.ptr, 4 * self._out.size, self._st.raw), "d2h")
        self._st.sync()
        self._queued = False
        return self._out.copy()

    def __del__(self) -> None:
        try:
            if self._p:
                if self._queued:
                    self._st.sync()
                self._l.dr_host_free(self._p)
                self._p = C.c_void_p()
        except Exception:
            pass


class ExtBuf:
    """Device memory owned by someone else (for example a torch tensor), seen through DevBuf's interface."""

    def __init__(self, ptr: int, nbytes: int, keep=None) -> None:
        self._ptr, self.nbytes, self._keep = int(ptr), int(nbytes), keep

    @property
    def ptr(self) -> int:
        return self._ptr

    def at(self, byte_offset: int) -> C.c_void_p:
        return C.c_void_p(self._ptr + int(byte_offset))

    def free(self) -> None:
        self._keep = None
