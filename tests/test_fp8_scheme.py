"""The arithmetic of the block-FP8 prefill, restated in numpy and held against the fp64 expert on the CPU.

Every E4M3 weight is an fp16 number, so the weight operand is exact. bf16 token rows become fp16 rows (a row whose largest magnitude
lies outside [2^-4, 2^15) is divided by a power of two first, which comes back after the gate/up product); each 128 inputs are summed
by themselves and the sum is multiplied by the block's scale in fp32; the SwiGLU intermediate is fp16. The kernel itself is compared with
the same fp64 expert in tests/test_gpu_fp8.py and tests/test_gpu_prefill_edges.py."""

from __future__ import annotations

import numpy as np
import pytest

from drama_rs_b200 import synth
from oracle import moe_oracle as orc

E4M3 = synth.e4m3_values()


def test_every_e4m3_number_is_an_fp16_number():
    v = E4M3[np.isfinite(E4M3)]
    assert len(v) == 254 and np.array_equal(v.astype(np.float16).astype(np.float32), v)


def fp16_rows(x: np.ndarray) -> tuple[np.ndarray, np.ndarray]:
    """The rows as fp16 and the power of two that each was divided by."""
    m = np.abs(x).max(axis=1)
    fac = np.where((m > 0) & ((m < 2.0**-4) | (m >= 2.0**15)), 2.0 ** np.floor(np.log2(np.where(m > 0, m, 1.0))), 1.0)
    return (x / fac[:, None]).astype(np.float16).astype(np.float64), fac


def product(codes: np.ndarray, scales: np.ndarray, x: np.ndarray) -> np.ndarray:
    """x [n, K] times the block-FP8 matrix transposed: exact sums over 128 inputs, scaled and added in fp32."""
    r, k = codes.shape
    w = E4M3[codes].astype(np.float64)
    y = np.zeros((x.shape[0], r), dtype=np.float32)
    for kb in range(k // 128):
        cols = slice(128 * kb, 128 * kb + 128)
        y += np.repeat(scales[:, kb], 128)[None].astype(np.float32) * (x[:, cols] @ w[:, cols].T).astype(np.float32)
    return y


@pytest.mark.parametrize("spread", [1.0, 100.0])
def test_scheme_against_the_fp64_expert(spread):
    host = synth.make_fp8_experts(21, synth.MoeShape(experts=2))
    rng = np.random.Generator(np.random.PCG64(81))
    for k in ("moe.gate_up.fp8_s", "moe.down.fp8_s"):  # spread 100: block scales from 1e-6 to 1e-2
        host[k] = (host[k] * np.exp(rng.uniform(-np.log(spread), np.log(spread), size=host[k].shape))).astype(np.float32)
    rows = rng.standard_normal((6, 2048), dtype=np.float32) * np.array([1, 1, 3, 0, 0.004, 1], dtype=np.float32)[:, None]
    x = synth.bf16_bits_to_f32(synth.f32_to_bf16_bits(rows)).astype(np.float64)
    xh, fac = fp16_rows(x)
    assert fac[4] < 2.0**-5 and (fac[[0, 1, 2, 3, 5]] == 1.0).all()
    h = product(host["moe.gate_up.fp8"][1], host["moe.gate_up.fp8_s"][1], xh).astype(np.float64) * fac[:, None]
    g, u = h[:, :512], h[:, 512:]
    act = (g / (1.0 + np.exp(-g)) * u).astype(np.float16).astype(np.float64)
    y = product(host["moe.down.fp8"][1], host["moe.down.fp8_s"][1], act)
    ref = orc.expert_forward(host, 1, x, np.float64)
    assert not y[3].any() and not ref[3].any()
    live = [0, 1, 2, 5]  # row 4's intermediate is so small that fp16 holds it as subnormal numbers
    assert (np.linalg.norm(y - ref, axis=1)[live] <= 5e-4 * np.linalg.norm(ref, axis=1)[live]).all()
    assert np.linalg.norm(h[4] - product(host["moe.gate_up.fp8"][1], host["moe.gate_up.fp8_s"][1], x[4:5])) <= 1e-6 * np.linalg.norm(h[4])
