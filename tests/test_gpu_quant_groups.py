"""drb_quant_q4 where its estimates cannot decide: groups far from zero or with scales among fp16's last numbers (the candidates that clip most
win there), an outlier, nearly constant groups, and kinds side by side in one warp, whose four groups share their branches. Weights at a 16-byte
address and one float behind it (two loaders). Bit for bit against the converter's restatement; a group with a NaN or an infinity, whose codes
the converter leaves undefined, must not change its neighbours."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from drama_rs_b200 import ffi
from drama_rs_b200.gpu import DevBuf, Stream, launched
from oracle import quant_oracle as qo

pytestmark = pytest.mark.gpu
F = np.float32
KINDS = ["normal", "offset", "far", "outlier", "small", "flat"]


def values(kind: str, groups: int) -> np.ndarray:
    r = np.random.Generator(np.random.PCG64(groups))
    w = r.standard_normal((groups, 64), dtype=F)
    pick = np.arange(groups)[:, None]
    if kind == "mixed":
        each = np.stack([values(k, groups) for k in KINDS])
        return np.take_along_axis(each, r.integers(0, len(KINDS), (1, groups, 1)), axis=0)[0]
    if kind == "offset":
        return (w + F(10.0) ** (pick % 6 - 2).astype(F)).astype(F)
    if kind == "far":  # the min's last place is a part of the scale
        return (w * F(0.3) + F(1000)).astype(F)
    if kind == "outlier":
        w[:, 5] *= 40
        w[::2, 60] *= 40
    if kind == "small":
        return (w * F(10.0) ** (-5 - pick % 3).astype(F)).astype(F)
    if kind == "flat":
        w = np.repeat(np.where(pick % 3 == 0, 0, w[:, :1]).astype(F), 64, axis=1)
        w[1::3, 7] = np.nextafter(w[1::3, 7], F(9))
    return w


def quantise(w: np.ndarray, shift: int) -> tuple[np.ndarray, np.ndarray]:
    l, st = ffi.lib(), Stream()
    groups = len(w)
    dw, dq, dsm = DevBuf.from_array(np.concatenate([np.zeros(shift, F), w.reshape(-1)]), st), DevBuf(groups * 32 + 64), DevBuf(groups * 4 + 64)
    dq.fill(0xAA, st)
    dsm.fill(0xAA, st)
    launched(l.drb_quant_q4(dw.at(4 * shift), C.c_size_t(groups), dq.at(0), dsm.at(0), st.raw), "quant_q4")
    q, sm = dq.download(np.uint8, groups * 32 + 64, st), dsm.download(np.uint16, groups * 2 + 32, st)
    assert (q[groups * 32 :] == 0xAA).all() and (sm[groups * 2 :] == 0xAAAA).all()
    return q[: groups * 32].reshape(groups, 32), sm[: groups * 2].reshape(groups, 2)


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("kind", KINDS + ["mixed"])
@pytest.mark.parametrize("groups", [1, 31, 33, 4097])
def test_quant_q4(kind, groups, shift):
    w = values(kind, groups)
    want_q, want_sm = qo.quant_q4(w.reshape(1, 1, -1))
    q, sm = quantise(w, shift)
    assert np.array_equal(q, want_q.reshape(groups, 32)) and np.array_equal(sm, want_sm.view(np.uint16).reshape(groups, 2))


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_neighbours_of_a_group_that_is_not_finite(bad):
    w = values("normal", 257)
    want_q, want_sm = qo.quant_q4(w.reshape(1, 1, -1))
    hit = np.arange(257) % 5 == 2
    w[hit, np.arange(257)[hit] % 64] = bad
    q, sm = quantise(w, 0)
    assert np.array_equal(q[~hit], want_q.reshape(257, 32)[~hit]) and np.array_equal(sm[~hit], want_sm.view(np.uint16).reshape(257, 2)[~hit])
