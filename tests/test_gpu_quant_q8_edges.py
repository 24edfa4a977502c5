"""drb_quant_q8 against the converter's restatement, bit for bit: group counts around a warp's four and a block's 32, values whose quotients
lie on one half, groups below fp16's least scale and constant groups."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from drama_rs_b200 import ffi, synth
from drama_rs_b200.gpu import DevBuf, Stream, launched
from oracle import quant_oracle as qo

pytestmark = pytest.mark.gpu


def values(kind: str, groups: int) -> np.ndarray:
    r = np.random.Generator(np.random.PCG64(groups))
    w = r.standard_normal((groups, 128), dtype=np.float32)
    if kind == "bf16":
        return synth.bf16_bits_to_f32(synth.f32_to_bf16_bits(w * 0.02))
    if kind == "ties":  # scale 2^-6 exactly, every quotient a multiple of one half
        w = (np.clip(np.round(w * 64 * 2), -254, 254) / 128).astype(np.float32)
        w[:, 3] = 127 * 2.0**-6
        return w
    if kind == "constant":
        return np.broadcast_to(w[:, :1], (groups, 128)).copy()
    return (w * np.float32(10.0) ** np.arange(-10, 6, dtype=np.float32)[np.arange(groups) % 16, None]).astype(np.float32)


@pytest.mark.parametrize("kind", ["bf16", "ties", "constant", "scales"])
@pytest.mark.parametrize("groups", [1, 3, 4, 5, 31, 33, 4097])
def test_quant_q8(kind, groups):
    l, st = ffi.lib(), Stream()
    w = values(kind, groups)
    dw, dq, ds = DevBuf.from_array(w, st), DevBuf(groups * 128 + 64), DevBuf(groups * 2 + 64)
    dq.fill(0xAA, st)
    ds.fill(0xAA, st)
    launched(l.drb_quant_q8(dw.at(0), C.c_size_t(groups), dq.at(0), ds.at(0), st.raw), "quant_q8")
    want_q, want_s = qo.quant_q8(w)
    q, s = dq.download(np.int8, groups * 128 + 64, st), ds.download(np.uint16, groups + 32, st)
    assert np.array_equal(q[: groups * 128].reshape(groups, 128), want_q) and (q[groups * 128 :].view(np.uint8) == 0xAA).all()
    assert np.array_equal(s[:groups], want_s.view(np.uint16).reshape(-1)) and (s[groups:] == 0xAAAA).all()
