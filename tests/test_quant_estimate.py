"""The int4 quantiser tells most of its 24 candidates apart by an estimate of their errors (csrc/quant.cuh, `estimate2`). Restated in
numpy: the estimate must lie within the bound that the kernel allows it, for every candidate that the kernel takes it for; and the bound by
the group's two ends, by which it passes the second half of the candidates over, must hold for those."""

import numpy as np
import pytest

F = np.float32


def groups(kind: str) -> np.ndarray:
    r = np.random.Generator(np.random.PCG64(11))
    w = r.standard_normal((3000, 64), dtype=F)
    if kind == "bf16":
        return ((w * F(0.02)).view(np.uint32) & 0xFFFF0000).view(F)
    if kind == "grid":  # quotients on and beside one half
        return (np.round(w * 8) / 16).astype(F)
    if kind == "offset":  # far from zero: the min's last place is a part of the scale
        return (w + F(10.0) ** r.integers(-2, 4, (3000, 1)).astype(F)).astype(F)
    if kind == "outlier":
        w[:, 5] *= 40
        return w
    return (w * F(10.0) ** r.integers(-9, 5, (3000, 1)).astype(F)).astype(F)


@pytest.mark.parametrize("kind", ["bf16", "grid", "offset", "outlier", "scales"])
def test_estimate_within_its_bound(kind):
    g = groups(kind)
    gmin, gmax = g.min(-1, keepdims=True), g.max(-1, keepdims=True)
    center = (gmin + gmax) * F(0.5)
    half, far = F(0.5) * (gmax - gmin)[:, 0], np.maximum(np.abs(gmin), np.abs(gmax))[:, 0]
    clip = np.maximum(F(0.2499) * half - F(2.0**-10) * (far + half) - F(1e-6), F(0)).astype(np.float64)
    assert (clip > 0).mean() > 0.15
    taken = 0
    for i in range(24):
        shrink = F(1.0 - 0.5 * i / 24)
        lo_c, hi_c = center + (gmin - center) * shrink, center + (gmax - center) * shrink
        with np.errstate(over="ignore", invalid="ignore"):
            scale = np.maximum(np.maximum((hi_c - lo_c) / F(15), F(1e-10)).astype(np.float16).astype(F), F(1e-10))
            lo = lo_c.astype(np.float16).astype(F)
            q = np.clip(np.rint((g - lo) / scale), 0, 15).astype(F)
            err = ((q * scale + lo - g) ** 2).astype(np.float64).sum(-1)
            if i >= 12:
                seen = np.isfinite(scale + lo)[:, 0]
                assert (err[seen] >= 1.99 * clip[seen] ** 2).all()
                continue
            # the hardware's reciprocal may be one unit off
            rcp = ((F(1) / scale).view(np.int32) + np.random.Generator(np.random.PCG64(i)).integers(-1, 2, scale.shape, dtype=np.int32)).view(F)
            # fused operations: exact in 64 bits for these magnitudes but for the last rounding
            mid = (-lo.astype(np.float64) * rcp - 7.5).astype(F)
            a = np.abs((g.astype(np.float64) * rcp + mid).astype(F))
        use = (a < 31).all(-1)
        taken += use.sum()
        r = (a[use] + F(32)).astype(F)
        n = np.minimum(((r.view(np.uint32) & 0xFFFC0000) | 0x00020000).view(F), F(39.5))
        s = ((r - n).astype(np.float64) ** 2).sum(-1)
        sc, eta = scale[use, 0].astype(np.float64), 2.0**-15 + 2.0**-21 * np.abs(lo[use, 0] * rcp[use, 0]).astype(np.float64)
        off = sc**2 * (17 * eta * np.sqrt(s) + 70 * eta**2 + 2.0**-16 * s) + 1e-42
        assert (np.abs(sc**2 * s - err[use]) <= off).all()
    assert taken > 12 * 3000 * (0.2 if kind in ("offset", "scales") else 0.9)
