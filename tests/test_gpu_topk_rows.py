"""dr_moe_topk at the edges of its blocks of four rows: one row, odd rows, a stride beyond E + 1, one to 256 experts, k up to 32, and ties, which
go to the lower index. Against a float64 softmax; the selection is exact."""

from __future__ import annotations

import numpy as np
import pytest

from drama_rs_b200 import ffi
from drama_rs_b200.gpu import DevBuf, Stream, launched

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("experts,topk", [(1, 1), (8, 8), (31, 3), (33, 32), (256, 8), (256, 32)])
@pytest.mark.parametrize("rows", [1, 3, 4, 5, 130])
def test_rows(rows, experts, topk):
    st, stride = Stream(), experts + 4
    rng = np.random.Generator(np.random.PCG64(rows + experts))
    logits = rng.standard_normal((rows, stride), dtype=np.float32) * 2
    logits[0, : experts // 2 + 1] = np.float32(1.5)  # equal logits: the lower index first
    dl = DevBuf.from_array(logits, st)
    idx, wts, gate = DevBuf(rows * topk * 4), DevBuf(rows * topk * 4), DevBuf(rows * 4)
    launched(ffi.lib().dr_moe_topk(dl.at(0), rows, experts, topk, stride, idx.at(0), wts.at(0), gate.at(0), st.raw), "topk")
    v = logits[:, :experts].astype(np.float64)
    want = np.argsort(-v, axis=1, kind="stable")[:, :topk]
    p = np.exp(np.take_along_axis(v, want, axis=1))
    got = wts.download(np.float32, rows * topk, st).reshape(rows, topk)
    assert np.array_equal(idx.download(np.int32, rows * topk, st).reshape(rows, topk), want)
    # a sum of up to 32 fp32 terms and three roundings, of exponentials good to two units
    assert np.abs(got / (p / p.sum(axis=1, keepdims=True)) - 1).max() <= 40 * 2.0**-24
    assert np.array_equal(gate.download(np.float32, rows, st), logits[:, experts])


@pytest.mark.parametrize("experts,topk,few", [(256, 8, 4), (256, 4, 1), (128, 4, 64), (96, 3, 2), (64, 24, 64), (32, 8, 64), (32, 32, 5), (9, 6, 1)])
def test_a_rows_routing_does_not_depend_on_the_batch(experts, topk, few):
    """Few rows and many may take different kernels: the same bits either way."""
    st, rows = Stream(), 4097
    rng = np.random.Generator(np.random.PCG64(experts + topk))
    logits = rng.standard_normal((rows, experts + 1), dtype=np.float32) * 2
    logits[1::3, : experts // 2] = np.float32(0.5)
    dl = DevBuf.from_array(logits, st)
    got = []
    for n in (few, rows):
        idx, wts, gate = DevBuf(rows * topk * 4), DevBuf(rows * topk * 4), DevBuf(rows * 4)
        launched(ffi.lib().dr_moe_topk(dl.at(0), n, experts, topk, experts + 1, idx.at(0), wts.at(0), gate.at(0), st.raw), "topk")
        got.append([idx.download(np.int32, few * topk, st), wts.download(np.uint32, few * topk, st), gate.download(np.uint32, few, st)])
    for a, b in zip(*got):
        assert np.array_equal(a, b)
