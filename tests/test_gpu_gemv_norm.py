"""dr_gemv_bf16 with a norm against float64: 1 / rms joins at the outputs, so inputs far from one are in. Rows around a warp's and a block's share."""

from __future__ import annotations

import numpy as np
import pytest

from drama_rs_b200 import ffi, synth
from drama_rs_b200.gpu import DevBuf, Stream, launched
from oracle import moe_oracle as orc

pytestmark = pytest.mark.gpu
K = 2048


@pytest.mark.parametrize("scale", [1e-3, 1.0, 1e3])
@pytest.mark.parametrize("n", [1, 16, 257, 4097])
def test_gemv_bf16(n, scale):
    l, st = ffi.lib(), Stream()
    r = np.random.Generator(np.random.PCG64(n))
    w = synth.f32_to_bf16_bits(r.standard_normal((n, K), dtype=np.float32) * np.float32(0.02))
    x = (r.standard_normal(K) * scale).astype(np.float32)
    x[5] = 30 * scale
    nw = (1 + 0.1 * r.standard_normal(K)).astype(np.float32)
    eps = 1e-6
    dw, dx, dnw = (DevBuf.from_array(a, st) for a in (w, x, nw))
    dy = DevBuf((n + 32) * 4)
    dy.fill(0xAA, st)
    for res in range(3):  # again at once: the launch before may still run
        launched(l.dr_gemv_bf16(dw.at(0), dx.at(0), dy.at(0), n, K, dnw.at(0), eps, None, 0, st.raw), "gemv_bf16")
    y = dy.download(np.float32, n + 32, st)
    assert (y[n:].view(np.uint32) == 0xAAAAAAAA).all()
    xn = x.astype(np.float64) * nw / np.sqrt((x.astype(np.float64) ** 2).mean() + eps)
    terms = synth.bf16_bits_to_f32(w).astype(np.float64) * xn
    # a lane sums 64 products in four chains, the lanes are folded in five steps; the product with nw, 1 / rms and its product come on top
    bound = (16 + 2 + 5 + 8) * 2.0**-24 * np.abs(terms).sum(axis=1)
    assert (np.abs(y[:n] - terms.sum(axis=1)) <= bound).all()
    assert np.abs(y[:n] - orc.gemv_bf16(w, xn, dtype=np.float64)).max() <= 2e-6 * np.abs(terms.sum(axis=1)).max() + 1e-7
