"""The int4 quantiser tells most of its 24 candidates apart by an estimate of their errors (csrc/quant.cuh, `estimate2`). Restated in
numpy: the estimate must lie within the bound that the kernel allows it, for every candidate that the kernel takes it for; and the bound by
the group's two ends, by which it passes the second half of the candidates over, must hold for those. The numbers are the kernel's own, read from
its source; that the kernel uses them as written here is for the bit-exact tests on the GPU."""

import os
import re

import numpy as np
import pytest

F = np.float32
with open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "drama_rs_b200", "csrc", "quant.cuh")) as _f:
    SRC = _f.read()


def numbers(line: str) -> list[float]:
    """The numbers that stand where `line` has @ in the source, which must have exactly one such place."""
    found = re.findall(re.escape(line).replace("@", r"((?:0x)?[0-9A-Fa-f.]+(?:p-?[0-9]+)?(?:e-?[0-9]+)?)[fu]*"), SRC)
    assert len(found) == 1, (line, found)
    found = found[0] if isinstance(found[0], tuple) else found
    return [float.fromhex(n) if n.startswith("0x") else float(n.rstrip("f")) for n in found]


LIGHT = int(numbers("Q4_LIGHT = @;")[0])
BASE, (MASK, HALF), (TOP,) = numbers("EST_BASE = @;")[0], [int(n) for n in numbers("EST_MASK = @, EST_HALF = @;")], numbers("EST_HALF)), EST_BASE + @);\n  const float q1")
ETA, ETA_MIN = numbers("eta = @ + @ * fabsf(c.lo) * c.rcp")
CUT, CUT1 = numbers("a0 < @ && a1 < @ ?")
BY_ROOT, BY_ETA, BY_SUM, LEAST = numbers("off = s2 * (@ * eta * root + @ * eta * eta + @ * s) + @;")
CLIP, CLIP_FAR, CLIP_LESS = numbers("clip = @ * half - @ * (far + half) - @;")
ENDS = numbers("clip > 0.f && @ * clip * clip >= bound")[0]


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
    clip = np.maximum(F(CLIP) * half - F(CLIP_FAR) * (far + half) - F(CLIP_LESS), F(0)).astype(np.float64)
    assert (clip > 0).mean() > 0.15
    taken = 0
    for i in range(24):
        shrink = F(1.0 - 0.5 * i / 24)
        lo_c, hi_c = center + (gmin - center) * shrink, center + (gmax - center) * shrink
        with np.errstate(over="ignore", invalid="ignore"):
            scale = np.maximum(np.maximum((hi_c - lo_c) / F(15), F(1e-10)).astype(np.float16).astype(F), F(1e-10))
            lo = lo_c.astype(np.float16).astype(F)
            q = np.clip(np.rint((g - lo) / scale), 0, 15).astype(F)
            off_by = q * scale + lo - g
            err = (off_by**2).astype(np.float64).sum(-1)
            if i >= LIGHT:  # the two ends' terms alone
                seen = np.isfinite(scale + lo)[:, 0]
                ends = np.take_along_axis(off_by, np.stack((g.argmin(-1), g.argmax(-1)), axis=-1), axis=-1).astype(np.float64)
                assert ((ends[seen] ** 2).sum(-1) >= ENDS * clip[seen] ** 2).all()
                continue
            # the hardware's reciprocal may be one unit off
            rcp = ((F(1) / scale).view(np.int32) + np.random.Generator(np.random.PCG64(i)).integers(-1, 2, scale.shape, dtype=np.int32)).view(F)
            # fused operations: exact in 64 bits for these magnitudes but for the last rounding
            mid = (-lo.astype(np.float64) * rcp - 7.5).astype(F)
            a = np.abs((g.astype(np.float64) * rcp + mid).astype(F))
        use = (a < CUT).all(-1)
        taken += use.sum()
        r = (a[use] + F(BASE)).astype(F)
        n = np.minimum(((r.view(np.uint32) & np.uint32(MASK)) | np.uint32(HALF)).view(F), F(BASE + TOP))
        s = ((r - n).astype(np.float64) ** 2).sum(-1)
        sc, eta = scale[use, 0].astype(np.float64), ETA + ETA_MIN * np.abs(lo[use, 0] * rcp[use, 0]).astype(np.float64)
        assert (np.abs(np.abs(r - n) - np.abs(off_by[use].astype(np.float64)) / sc[:, None]) <= eta[:, None]).all()  # input by input
        off = sc**2 * (BY_ROOT * eta * np.sqrt(s) + BY_ETA * eta**2 + BY_SUM * s) + LEAST
        assert (np.abs(sc**2 * s - err[use]) <= off).all()
    assert CUT == CUT1 and taken > LIGHT * 3000 * (0.2 if kind in ("offset", "scales") else 0.9)
