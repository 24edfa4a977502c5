"""drb_quant_q4 where a group's range is so small that its scale sits at the converter's floor of 1e-10 (below fp16's least number). The scale
has 24 bits there, so a quotient may round onto a boundary that the exact one misses: the division itself decides. Bit for bit against the
converter's restatement."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from drama_rs_b200 import ffi
from drama_rs_b200.gpu import DevBuf, Stream, launched
from oracle import quant_oracle as qo

pytestmark = pytest.mark.gpu


def values(kind: str, groups: int) -> np.ndarray:
    r = np.random.Generator(np.random.PCG64(groups))
    n = r.integers(0, 14, (groups, 64))
    w = ((n + 0.5) * 1e-10).astype(np.float32)  # on the boundaries between codes
    w[:, 0] = 0
    if kind == "beside":
        w = (w.view(np.int32) + r.integers(-1, 2, w.shape, dtype=np.int32) * (w != 0)).view(np.float32)
    if kind == "negative":
        w[:, 1::2] *= -1
    if kind == "offset":  # from a min that is one of fp16's smallest numbers
        w += (np.float32(2.0**-24) * r.integers(-4, 5, (groups, 1))).astype(np.float32)
    if kind == "spans":
        w = (r.standard_normal((groups, 64), dtype=np.float32) * np.float32(10.0) ** r.uniform(-12, -6, (groups, 1)).astype(np.float32)).astype(np.float32)
    return w


@pytest.mark.parametrize("kind", ["ties", "beside", "negative", "offset", "spans"])
@pytest.mark.parametrize("groups", [1, 33, 4097])
def test_quant_q4(kind, groups):
    l, st = ffi.lib(), Stream()
    w = values(kind, groups)
    dw, dq, dsm = DevBuf.from_array(w, st), DevBuf(groups * 32), DevBuf(groups * 4)
    launched(l.drb_quant_q4(dw.at(0), C.c_size_t(groups), dq.at(0), dsm.at(0), st.raw), "quant_q4")
    want_q, want_sm = qo.quant_q4(w.reshape(1, 1, -1))
    assert np.array_equal(dq.download(np.uint8, groups * 32, st), want_q.reshape(-1))
    assert np.array_equal(dsm.download(np.uint16, groups * 2, st), want_sm.view(np.uint16).reshape(-1))
