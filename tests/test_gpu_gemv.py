"""Dense GEMVs through the C ABI against the oracle."""

import ctypes as C
import os

import numpy as np
import pytest

from drama_rs_b200 import ffi, synth
from drama_rs_b200.gpu import DevBuf, Stream, launched
from oracle import moe_oracle as orc
from tests.helpers import NULL, device_error_word

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def st():
    return Stream()


def run_q8(st, q, s, x, res=None, nw=None, eps=1e-6, alias=False):
    l = ffi.lib()
    n, k = q.shape
    dq, ds, dx = DevBuf.from_array(q, st), DevBuf.from_array(s, st), DevBuf.from_array(x, st)
    dy = DevBuf(n * 4)
    dy.fill(0xFF, st)
    dres = None
    if res is not None:
        if alias:
            dy.upload(res, st)
            dres = dy
        else:
            dres = DevBuf.from_array(res, st)
    dnw = DevBuf.from_array(nw, st) if nw is not None else None
    rc = l.dr_gemv_q8(dq.at(0), ds.at(0), dx.at(0), dres.at(0) if dres else NULL, dy.at(0), n, k,
                      dnw.at(0) if dnw else NULL, eps, NULL, 0, st.raw)
    if rc != 0:
        return rc
    launched(rc, "gemv_q8")
    return dy.download(np.float32, n, st)


@pytest.mark.parametrize("n,k", [(4096, 2048), (2048, 4096), (8192, 2048), (64, 512), (2048, 512), (37, 2048), (4097, 2048),
                                 (300, 6144), (129, 8192), (1, 2048)])
def test_gemv_q8_shapes(st, n, k):
    q, s = synth.make_q8(n * 7 + k, n, k)
    x = synth.make_x(n + k, 1, k)[0]
    y = run_q8(st, q, s, x)
    ref = orc.gemv_q8(q, s, x, dtype=np.float64)
    scale = np.abs(ref).max()
    # activations enter as four 7-bit limbs per value (2^-28 of the largest of 128): about 1e-7 of the output scale, fp32 sums and scales
    assert np.abs(y - ref).max() <= 1e-5 * scale + 5e-6, (n, k)
    assert device_error_word() == 0


def test_gemv_q8_golden_and_bf16_cast(st, golden_dir):
    g = np.load(os.path.join(golden_dir, "gemv_q8.npz"))
    for j, (n, k) in enumerate([(4096, 2048), (2048, 4096), (8192, 2048), (151936, 2048)]):
        q, s = synth.make_q8(100 + j, n, k)
        x = synth.make_x(100 + j, 1, k)[0]
        y = run_q8(st, q, s, x)
        step = max(1, n // 4096)
        ref64 = g[f"y64_{n}_{k}"]
        assert np.abs(y[::step] - ref64).max() <= 2e-6 * np.abs(ref64).max()
        # cast to bf16 as the benchmark configuration asks: at most one bf16 ulp from the cast of the fp64 result
        yb = orc.f32_to_bf16_bits(y[::step]).astype(np.int32)
        rb = orc.f32_to_bf16_bits(ref64.astype(np.float32)).astype(np.int32)
        assert np.abs(yb - rb).max() <= 1


def test_gemv_q8_residual_alias_and_norm(st):
    n, k = 2048, 4096
    q, s = synth.make_q8(5, n, k)
    x = synth.make_x(6, 1, k)[0]
    res = synth.make_x(7, 1, n)[0]
    nw = (1.0 + 0.1 * synth.make_x(8, 1, k)[0]).astype(np.float32)
    ref = orc.gemv_q8(q, s, x, res=res, nw=nw, eps=1e-6, dtype=np.float64)
    for alias in (False, True):
        y = run_q8(st, q, s, x, res=res, nw=nw, alias=alias)
        assert np.abs(y - ref).max() <= 2e-6 * np.abs(ref).max()


def test_gemv_q8_rejects_unsupported_k(st):
    q, s = synth.make_q8(1, 16, 1024)
    assert run_q8(st, q, s, np.zeros(1024, np.float32)) == -1


@pytest.mark.parametrize("i,k", [(512, 2048), (1536, 2048), (100, 4096)])
def test_gemv_q8_swiglu(st, i, k):
    l = ffi.lib()
    q, s = synth.make_q8(i + k, 2 * i, k)
    x = synth.make_x(i, 1, k)[0]
    nw = (1.0 + 0.1 * synth.make_x(9, 1, k)[0]).astype(np.float32)
    dq, ds, dx, dnw = (DevBuf.from_array(a, st) for a in (q, s, x, nw))
    dy = DevBuf(i * 4)
    launched(l.dr_gemv_q8_swiglu(dq.at(0), ds.at(0), dx.at(0), dy.at(0), i, k, dnw.at(0), 1e-6, NULL, 0, st.raw), "swiglu")
    y = dy.download(np.float32, i, st)
    ref = orc.gemv_q8_swiglu(q, s, x, i, nw=nw, eps=1e-6, dtype=np.float64)
    assert np.abs(y - ref).max() <= 4e-6 * np.abs(ref).max()


@pytest.mark.parametrize("n", [4097, 257, 16])
def test_gemv_bf16(st, n):
    l = ffi.lib()
    rng = np.random.Generator(np.random.PCG64(n))
    w = synth.f32_to_bf16_bits(rng.standard_normal((n, 2048), dtype=np.float32) * np.float32(0.02))
    x = synth.make_x(n, 1, 2048)[0]
    dw, dx = DevBuf.from_array(w, st), DevBuf.from_array(x, st)
    dy = DevBuf(n * 4)
    # prefetch arguments pointing at a real region must be harmless
    launched(l.dr_gemv_bf16(dw.at(0), dx.at(0), dy.at(0), n, 2048, NULL, 0.0, C.cast(dw.at(0), C.c_void_p), w.nbytes, st.raw), "gemv_bf16")
    y = dy.download(np.float32, n, st)
    ref = orc.gemv_bf16(w, x, dtype=np.float64)
    assert np.abs(y - ref).max() <= 2e-6 * np.abs(ref).max() + 1e-7
    assert l.dr_gemv_bf16(dw.at(0), dx.at(0), dy.at(0), n, 1024, NULL, 0.0, NULL, 0, st.raw) == -1


def test_gemv_q8_extreme_codes_against_a_constant_slice(st):
    """Every code at -128 against a slice of equal negative activations: each 16-byte chunk's integer sum reaches
    16 * 128 * 2^20 = 2^31, one past what an int32 recombination of the limbs can hold."""
    n, k = 64, 2048
    q = np.full((n, k), -128, dtype=np.int8)
    q[1::2] = 127
    s = np.full((n, k // 128), 0.01, dtype=np.float16)
    x = np.full(k, -1.5, dtype=np.float32)
    y = run_q8(st, q, s, x)
    ref = orc.gemv_q8(q, s, x, dtype=np.float64)
    assert np.abs(y - ref).max() <= 1e-5 * np.abs(ref).max(), (y[:4], ref[:4])
    assert device_error_word() == 0


@pytest.mark.parametrize("k", [512, 2048, 4096, 6144, 8192])
@pytest.mark.parametrize("n", [1, 15, 17, 148 * 16 + 5, 148 * 64 + 77])
def test_gemv_q8_tile_edges(st, n, k):
    """Row counts around the sixteen-row tiles, the 64-row batches and the ring of stages, with norm and aliased residual."""
    if n * k > 40_000_000:
        n = 148 * 17 + 9
    q, s = synth.make_q8(n + k, n, k)
    rng = np.random.Generator(np.random.PCG64(n * k))
    x = synth.make_x(n + 3 * k, 1, k)[0]
    x[rng.integers(0, k, 8)] *= 300.0  # outliers share their group of 128 with ordinary inputs
    nw = (1.0 + 0.1 * rng.standard_normal(k)).astype(np.float32)
    res = rng.standard_normal(n).astype(np.float32)
    y = run_q8(st, q, s, x, res=res, nw=nw, alias=True)
    xn = orc.rmsnorm(x[None].astype(np.float64), nw, 1e-6, np.float64)[0]
    ref = orc.gemv_q8(q, s, xn, dtype=np.float64) + res
    assert np.abs(y - ref).max() <= 1e-5 * np.abs(ref).max() + 5e-6, (n, k)
    assert device_error_word() == 0
