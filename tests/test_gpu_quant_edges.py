"""drb_quant_q4 against the converter's restatement: group counts around a block's 32, and values that sit on rounding
boundaries (bf16 grids), span one constant, or lie far from 1."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from drama_rs_b200 import ffi, synth
from drama_rs_b200.gpu import DevBuf, Stream, launched
from oracle import quant_oracle as qo

pytestmark = pytest.mark.gpu


def values(kind: str, groups: int) -> np.ndarray:
    w = np.random.Generator(np.random.PCG64(groups)).standard_normal((groups, 64), dtype=np.float32)
    if kind == "bf16":
        return synth.bf16_bits_to_f32(synth.f32_to_bf16_bits(w * 0.02))
    if kind == "grid":  # quotients on and beside one half
        return (np.round(w * 8) / 16).astype(np.float32)
    if kind == "constant":
        return np.broadcast_to(w[:, :1] * 300, (groups, 64)).copy()
    return (w * np.float32(10.0) ** np.arange(-6, 6, dtype=np.float32)[np.arange(groups) % 12, None]).astype(np.float32)


@pytest.mark.parametrize("kind", ["bf16", "grid", "constant", "scales"])
@pytest.mark.parametrize("groups", [1, 31, 33, 4097])
def test_quant_q4(kind, groups):
    l, st = ffi.lib(), Stream()
    w = values(kind, groups)
    dw, dq, dsm = DevBuf.from_array(w, st), DevBuf(groups * 32 + 64), DevBuf(groups * 4)
    want_q, want_sm = qo.quant_q4(w.reshape(1, 1, -1))
    for shift in (0, 1):  # codes at any address
        dq.fill(0xAA, st)
        launched(l.drb_quant_q4(dw.at(0), C.c_size_t(groups), dq.at(shift), dsm.at(0), st.raw), "quant_q4")
        q = dq.download(np.uint8, groups * 32 + 64, st)
        assert np.array_equal(q[shift : shift + groups * 32], want_q.reshape(-1)) and (q[shift + groups * 32 :] == 0xAA).all()
        assert np.array_equal(dsm.download(np.uint16, groups * 2, st), want_sm.view(np.uint16).reshape(-1))
