"""The grouped prefill GEMMs at the edges of their tiles: token boxes of eight, MMA columns of sixteen, items of 64 (int4)
and 32 (FP8) tokens, the array's first rows, more experts than one launch takes, and the gathered form behind the
peer-store entry point."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from drama_rs_b200 import ffi, synth
from drama_rs_b200.engine import MoePrefill
from drama_rs_b200.gpu import DevBuf, Stream, launched
from drama_rs_b200.model import Fp8Experts, MoeLayer
from oracle import moe_oracle as orc
from tests.helpers import NULL, device_error_word

pytestmark = pytest.mark.gpu

EDGES = {
    "boxes": [1, 2, 3, 4, 5, 7, 8, 9, 12, 15, 16, 17, 23, 24, 25, 0],
    "items": [31, 32, 33, 63, 64, 65, 0, 127, 128, 129, 1, 0, 40, 47, 48, 49],
    "first rows": [0, 3, 0, 2, 1, 0, 0, 9, 0, 0, 0, 0, 0, 0, 0, 6],
    "one row": [0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 1, 0, 0, 0, 0],
}


@pytest.fixture(scope="module")
def st():
    return Stream()


def check_rows(y, host, x, counts, offsets, experts, bar=8e-4):
    assert device_error_word() == 0
    for e, c, o in zip(experts, counts, offsets):
        if c:
            ref = orc.expert_forward(host, e, x[o : o + c], np.float64)
            rel = np.linalg.norm(y[o : o + c] - ref, axis=1) / np.linalg.norm(ref, axis=1)
            assert np.isfinite(rel).all() and rel.max() <= bar, (e, c, float(rel.max()))


def run_groups(st, fmt, host, xb, counts, offsets):
    """dr_moe_prefill or dr_moe_prefill_fp8 over bf16 rows sorted by expert."""
    l, n, e = ffi.lib(), len(xb), len(counts)
    dxp, dcnt, doff = DevBuf.from_array(xb, st), DevBuf.from_array(counts, st), DevBuf.from_array(offsets, st)
    dact, dy = DevBuf(n * 1024), DevBuf(n * 8192)
    dy.fill(0xFF, st)
    if fmt == "int4":
        dev = MoeLayer.upload(host, st)
        w, call = (*dev.gate_up.expert(0), *dev.down.expert(0)), l.dr_moe_prefill
    else:
        f8 = Fp8Experts.upload(host, st)
        w, call = (f8.gu_w.at(0), f8.gu_s.at(0), f8.d_w.at(0), f8.d_s.at(0)), l.dr_moe_prefill_fp8
    launched(call(*w, dxp.at(0), doff.at(0), dcnt.at(0), dact.at(0), dy.at(0), e, 2048, 512, st.raw), "prefill")
    return dy.download(np.float32, n * 2048, st).reshape(n, 2048)


def make_groups(edge, fmt):
    host = (synth.make_layer if fmt == "int4" else synth.make_fp8_experts)(31, synth.MoeShape(experts=16))
    counts = np.array(EDGES[edge], dtype=np.int32)
    n = int(counts.sum())
    return host, counts, (np.cumsum(counts) - counts).astype(np.int32), np.random.Generator(np.random.PCG64(n)).standard_normal((n, 2048), dtype=np.float32)


@pytest.mark.parametrize("fmt", ["int4", "fp8"])
@pytest.mark.parametrize("edge", EDGES)
def test_group_sizes(st, fmt, edge):
    host, counts, offsets, xf = make_groups(edge, fmt)
    xb = synth.f32_to_bf16_bits(xf)
    y = run_groups(st, fmt, host, xb, counts, offsets)
    check_rows(y, host, synth.bf16_bits_to_f32(xb).astype(np.float64), counts, offsets, range(16))


@pytest.mark.parametrize("fmt", ["int4", "fp8"])
@pytest.mark.parametrize("edge", ["boxes", "items", "first rows", "one row"])
def test_rows_divided_by_a_power_of_two(st, fmt, edge):
    """bf16 rows whose largest magnitude leaves [2^-4, 2^15) are divided by a power of two on their way to fp16 and multiplied back behind the
    gate/up product: every second expert gets rows far below the range, the others rows with one value far above it. Each row
    has a power of its own. The experts' scales are moved so that the fp16 intermediate stays in its range, and every row is compared."""
    host, counts, offsets, xf = make_groups(edge, fmt)
    rng = np.random.Generator(np.random.PCG64(3))
    name = "moe.gate_up.sm" if fmt == "int4" else "moe.gate_up.fp8_s"
    host[name] = host[name].copy()
    for e in range(16):
        rows = slice(offsets[e], offsets[e] + counts[e])
        if e % 2:
            host[name][e] *= 64.0 if fmt == "int4" else 256.0
            xf[rows] *= 2.0 ** -rng.integers(8, 11, (counts[e], 1))
        else:
            host[name][e] *= 2.0**-6 if fmt == "int4" else 2.0**-4
            xf[np.arange(offsets[e], offsets[e] + counts[e]), rng.integers(0, 2048, counts[e])] = 2.0 ** rng.integers(15, 17, counts[e])
    xb = synth.f32_to_bf16_bits(xf)
    x = synth.bf16_bits_to_f32(xb).astype(np.float64)
    top = np.abs(x).max(axis=1)
    assert ((top < 2.0**-4) | (top >= 2.0**15)).all()
    # one large value carries its row, so that its weight's rounding to fp16 does not average out: the steps restated in numpy
    # measure 6.1e-4 (int4) and 3.3e-4 (FP8) for the worst row
    check_rows(run_groups(st, fmt, host, xb, counts, offsets), host, x, counts, offsets, range(16), bar=1e-3)


@pytest.mark.parametrize("fmt", ["int4", "fp8"])
@pytest.mark.parametrize("edge", EDGES)
def test_extreme_rows_stay_finite(st, fmt, edge):
    """Rows whose activations leave fp16 altogether: clamped, or rounded to nothing, but finite; the rows beside them are right."""
    host, counts, offsets, xf = make_groups(edge, fmt)
    n = len(xf)
    xf[0] *= 1e6
    xf[n - 1] *= 1e-6 if n > 1 else 1.0
    xb = synth.f32_to_bf16_bits(xf)
    y = run_groups(st, fmt, host, xb, counts, offsets)
    assert np.isfinite(y).all()
    x = synth.bf16_bits_to_f32(xb).astype(np.float64)
    for e in range(16):
        rows = [r for r in range(offsets[e], offsets[e] + counts[e]) if 0 < r < n - 1]
        if rows:
            check_rows(y[rows], host, x[rows], [len(rows)], [0], [e])
    assert device_error_word() == 0


def test_more_experts_than_one_launch_takes(st):
    import torch

    l, e = ffi.lib(), 1027
    g = torch.Generator(device="cuda").manual_seed(5)
    q = [torch.randint(0, 256, (e, n, k // 2), dtype=torch.uint8, device="cuda", generator=g) for n, k in ((1024, 2048), (2048, 512))]
    s = [(torch.randn((e, n, k // 64), device="cuda", generator=g) * 0.01).abs().clamp_min(1e-4).half() for n, k in ((1024, 2048), (2048, 512))]
    sm = [torch.stack((v, (v.float() * -8.0).half()), dim=-1).contiguous() for v in s]
    hit = {0: 5, 511: 17, 1023: 3, 1024: 9, 1026: 66}
    counts = np.zeros(e, dtype=np.int32)
    counts[list(hit)] = list(hit.values())
    offsets = (np.cumsum(counts) - counts).astype(np.int32)
    n = int(counts.sum())
    xb = synth.f32_to_bf16_bits(np.random.Generator(np.random.PCG64(8)).standard_normal((n, 2048), dtype=np.float32))
    dxp, dcnt, doff = DevBuf.from_array(xb, st), DevBuf.from_array(counts, st), DevBuf.from_array(offsets, st)
    dact, dy = DevBuf(n * 1024), DevBuf(n * 8192)
    torch.cuda.synchronize()
    p = lambda t: C.c_void_p(t.data_ptr())
    launched(l.dr_moe_prefill(p(q[0]), p(sm[0]), p(q[1]), p(sm[1]), dxp.at(0), doff.at(0), dcnt.at(0), dact.at(0), dy.at(0), e, 2048, 512, st.raw), "prefill")
    y = dy.download(np.float32, n * 2048, st).reshape(n, 2048)
    x = synth.bf16_bits_to_f32(xb).astype(np.float64)
    names = ("moe.gate_up.q4", "moe.down.q4", "moe.gate_up.sm", "moe.down.sm")
    for ex in hit:
        host = {k: t[ex : ex + 1].cpu().numpy() for k, t in zip(names, (*q, *sm))}
        check_rows(y[offsets[ex] : offsets[ex] + counts[ex]], host, x[offsets[ex] : offsets[ex] + counts[ex]], [counts[ex]], [0], [0])


@pytest.mark.parametrize("rows", [1, 5, 40])
def test_gathered_rows_and_stored_results(st, rows):
    """drb_moe_prefill_block_peers with one rank: its own buffer is the peer. Same results as drb_moe_prefill_block."""
    l, shape = ffi.lib(), synth.MoeShape(experts=16)
    dev = MoeLayer.upload(synth.make_layer(32, shape), st)
    rng = np.random.Generator(np.random.PCG64(rows))
    xh = rng.standard_normal((rows, 2048), dtype=np.float32).astype(np.float16)
    idx = np.stack([rng.permutation(16)[:8] for _ in range(rows)]).astype(np.int32)
    n = rows * 8
    i32 = lambda m: DevBuf(m * 4)
    dx, didx = DevBuf.from_array(xh, st), DevBuf.from_array(idx, st)
    cnt, off, slot, row = i32(16), i32(16), i32(n), i32(n)
    launched(l.drb_moe_group(didx.at(0), rows, 8, 0, 16, cnt.at(0), off.at(0), slot.at(0), row.at(0), st.raw), "group")
    act, sh_act = DevBuf(n * 1024), DevBuf(rows * 1024)
    out = {}
    for name in ("block", "peers"):
        y, sh, dst = DevBuf(n * 8192), DevBuf(rows * 8192), DevBuf.from_array(np.arange(n, dtype=np.int32), st)
        w = (*dev.gate_up.expert(0), *dev.down.expert(0), *dev.shared_gate_up.rows(0), *dev.shared_down.rows(0))
        bufs = (dx.at(0), row.at(0), off.at(0), cnt.at(0), act.at(0), y.at(0), sh_act.at(0), sh.at(0), rows, 16, 2048, 512)
        if name == "block":
            launched(l.drb_moe_prefill_block(*w, *bufs, 1, NULL, st.raw), name)
            res = y
        else:
            res = DevBuf(n * 8192)
            table = DevBuf.from_array(np.array([res.ptr], dtype=np.uint64), st)
            launched(l.drb_moe_prefill_block_peers(*w, *bufs, dst.at(0), table.at(0), n, 0, st.raw), name)
        out[name] = (res.download(np.float32, n * 2048, st), sh.download(np.float32, rows * 2048, st))
    assert device_error_word() == 0
    for a, b in zip(out["block"], out["peers"]):
        assert np.linalg.norm(a - b) <= 2e-4 * np.linalg.norm(a)


@pytest.mark.parametrize("f16", [True, False], ids=["f16", "bf16"])
@pytest.mark.parametrize("rows,e1", [(1, 257), (15, 1), (16, 8), (17, 9), (40, 257), (2400, 257), (2400, 401)])
def test_router_logits_tiles(st, rows, e1, f16):
    """Row groups of 16, output tiles of 8, and more row groups than multiprocessors (all the tiles in one block, or in two)."""
    rng = np.random.Generator(np.random.PCG64(rows + e1))
    x = rng.standard_normal((rows, 2048), dtype=np.float32) * rng.choice([1e-3, 1.0, 30.0], (rows, 1)).astype(np.float32)
    xb = x.astype(np.float16) if f16 else synth.f32_to_bf16_bits(x)
    wb = synth.f32_to_bf16_bits(rng.standard_normal((e1, 2048), dtype=np.float32) * 0.02)
    bias = rng.standard_normal((rows, e1), dtype=np.float32)
    dx, dw, dl = DevBuf.from_array(xb, st), DevBuf.from_array(wb, st), DevBuf.from_array(bias, st)
    call = ffi.lib().drb_router_logits_f16 if f16 else ffi.lib().drb_router_logits
    launched(call(dx.at(0), dw.at(0), dl.at(0), rows, e1, 2048, 2.0, st.raw), "router_logits")
    wide = lambda bits: (bits.astype(np.uint32) << 16).view(np.float32).astype(np.float64)  # noqa: E731
    xv, wv = xb.astype(np.float64) if f16 else wide(xb), wide(wb)
    err = np.abs(dl.download(np.float32, rows * e1, st).reshape(rows, e1) - (xv @ wv.T + 2.0 * bias))
    assert (err <= 3e-7 * (np.abs(xv) @ np.abs(wv).T + 2.0 * np.abs(bias)) + 1e-9).all()


@pytest.mark.parametrize("experts,topk", [(256, 8), (40, 3), (8, 8)])
@pytest.mark.parametrize("rows", [1, 2, 16, 17, 32])
def test_few_rows_route_like_many(st, experts, topk, rows):
    """Up to 32 rows take one routing launch, more take two: weights, experts and results of a row are the same."""
    host = synth.make_layer(35, synth.MoeShape(experts=experts))
    dev = MoeLayer.upload(host, st)
    x = synth.make_x(36, 33, 2048)
    x[3] = x[2]  # equal rows, and ties between experts' logits in a row of zeros
    x[4] = 0.0
    few, many = MoePrefill(dev, rows, topk, st=st), MoePrefill(dev, 33, topk, st=st)
    y, ref = few.run(x[:rows]), many.run(x)
    assert device_error_word() == 0
    for name in ("idx", "wts"):
        a, b = (getattr(p, name).download(np.uint32, rows * topk, st) for p in (few, many))
        assert np.array_equal(a, b), name
    assert np.array_equal(few.sgate.download(np.uint32, rows, st), many.sgate.download(np.uint32, rows, st))
    idx = few.idx.download(np.int32, rows * topk, st)
    assert np.array_equal(few.counts.download(np.int32, experts, st), np.bincount(idx, minlength=experts))
    assert sorted(few.slot_of.download(np.int32, rows * topk, st)) == list(range(rows * topk))
    assert np.abs(y - ref[:rows]).max() <= 1e-6 * np.abs(ref).max()


@pytest.mark.parametrize("fmt", ["int4", "fp8"])
def test_results_at_any_float_and_refused_addresses(st, fmt):
    """y and sh_out may start at any float: same bits as at an aligned address, nothing written beside them. Rows, act and weights
    are read in 16-byte pieces: other addresses are refused before anything is launched."""
    l, shape = ffi.lib(), synth.MoeShape(experts=16)
    counts = np.array([1, 9, 0, 3, 17, 0, 2, 8, 0, 0, 5, 33, 1, 0, 4, 7], dtype=np.int32)
    offsets = (np.cumsum(counts) - counts).astype(np.int32)
    n = int(counts.sum())
    xb = synth.f32_to_bf16_bits(np.random.Generator(np.random.PCG64(4)).standard_normal((n, 2048), dtype=np.float32))
    dxp, dcnt, doff = DevBuf(n * 4096 + 16), DevBuf.from_array(counts, st), DevBuf.from_array(offsets, st)
    dxp.upload(xb, st)
    dact, shact = DevBuf(n * 1024 + 16), DevBuf(n * 1024 + 16)
    dev = MoeLayer.upload(synth.make_layer(33, shape), st)
    if fmt == "int4":
        shared = (*dev.shared_gate_up.rows(0), *dev.shared_down.rows(0))

        def call(y, sh=None, xp=dxp.at(0), act=dact.at(0), off=0):
            w = (C.c_void_p(dev.gate_up.q.ptr + off), dev.gate_up.sm.at(0), *dev.down.expert(0), *shared)
            return l.drb_moe_prefill_block(*w, xp, NULL, doff.at(0), dcnt.at(0), act, y, shact.at(0), sh, n, 16, 2048, 512, 0, NULL, st.raw)
    else:
        f8 = Fp8Experts.upload(synth.make_fp8_experts(33, shape), st)

        def call(y, sh=None, xp=dxp.at(0), act=dact.at(0), off=0):
            return l.dr_moe_prefill_fp8(f8.gu_w.at(off), f8.gu_s.at(0), f8.d_w.at(0), f8.d_s.at(0), xp, doff.at(0), dcnt.at(0), act, y, 16, 2048, 512, st.raw)

    words, got = n * 2048, {}
    dy, dsh = DevBuf(words * 4 + 32), DevBuf(words * 4 + 32)
    for at in (16, 4, 8, 12):
        dy.fill(0x55, st), dsh.fill(0x55, st)
        launched(call(dy.at(at), dsh.at(at)), "prefill")
        for name, buf in (("y", dy), ("shared", dsh)):
            raw = buf.download(np.uint32, words + 8, st)
            assert (raw[: at // 4] == 0x55555555).all() and (raw[at // 4 + words :] == 0x55555555).all(), (name, at)
            got.setdefault(name, raw[at // 4 : at // 4 + words])
            assert np.array_equal(raw[at // 4 : at // 4 + words], got[name]), (name, at)
    assert np.isfinite(got["y"].view(np.float32)).all() and device_error_word() == 0
    dy.fill(0x55, st)
    for bad in ({"xp": dxp.at(2)}, {"xp": dxp.at(8)}, {"act": dact.at(8)}, {"off": 8}):
        assert call(dy.at(0), dsh.at(0), **bad) == -3
    assert (dy.download(np.uint32, words, st) == 0x55555555).all() and l.dr_last_error() == 0


def test_layer_call_refuses_addresses_it_cannot_use(st):
    dev = MoeLayer.upload(synth.make_layer(34, synth.MoeShape(experts=16)), st)
    pre = MoePrefill(dev, 4, st=st)
    x = synth.make_x(37, 4, 2048)
    pre.x.upload(x, st)
    w, b = (a._obj for a in pre._layer_args())
    for struct, names in ((b, ("x", "rows16", "y", "sh_out", "act", "sh_act")), (w, ("router", "gu_q", "gu_sm", "d_q", "d_sm", "sgu_q", "sd_q"))):
        for name in names:
            p = getattr(struct, name)
            setattr(struct, name, p + 8)
            assert ffi.lib().drb_moe_prefill_layer(C.byref(w), C.byref(b), 4, 16, 8, 2048, 512, 1e-6, st.raw) == -3, name
            setattr(struct, name, p)
    assert np.array_equal(pre.x.download(np.float32, 4 * 2048, st).reshape(4, 2048), x) and ffi.lib().dr_last_error() == 0


@pytest.mark.parametrize("gathered", [False, True])
def test_gaps_between_the_experts_slots(st, gathered):
    """Offsets that leave gaps, and more experts than one preparing launch takes: the slots between the experts are nobody's. Their
    row_of is not looked at (it names a row of NaN here) and their rows of y keep what the caller had there."""
    l, e = ffi.lib(), 1026
    host = synth.make_layer(38, synth.MoeShape(experts=2))
    dev = MoeLayer.upload(host, st)
    counts, offsets = np.zeros(e, dtype=np.int32), np.zeros(e, dtype=np.int32)
    counts[[0, 1]], offsets[[0, 1]] = [3, 12], [2, 11]  # slots 0, 1, 5 .. 10 and from 23 on belong to no expert
    n, slots = 16, 30
    rng = np.random.Generator(np.random.PCG64(6))
    xf = rng.standard_normal((n, 2048), dtype=np.float32)
    xf[0] = np.nan
    row_of = np.zeros(slots, dtype=np.int32)
    own = np.r_[2:5, 11:23]
    row_of[own] = rng.permutation(15) + 1
    if not gathered:
        xf = np.where(np.isin(np.arange(slots), own)[:, None], xf[row_of], np.float32(np.nan))
    xb = synth.f32_to_bf16_bits(xf)
    dx, drow, dcnt, doff = (DevBuf.from_array(a, st) for a in (xb, row_of, counts, offsets))
    dact, dy, dsh = DevBuf(slots * 1024), DevBuf(slots * 8192), DevBuf(16)
    dy.fill(0x55, st)
    w = (*dev.gate_up.expert(0), *dev.down.expert(0))
    if gathered:
        rc = l.drb_moe_prefill_block(*w, *dev.shared_gate_up.rows(0), *dev.shared_down.rows(0), dx.at(0), drow.at(0), doff.at(0), dcnt.at(0), dact.at(0),
                                     dy.at(0), dact.at(0), dsh.at(0), 0, e, 2048, 512, 0, NULL, st.raw)
    else:
        rc = l.dr_moe_prefill(*w, dx.at(0), doff.at(0), dcnt.at(0), dact.at(0), dy.at(0), e, 2048, 512, st.raw)
    launched(rc, "prefill")
    raw = dy.download(np.uint32, slots * 2048, st).reshape(slots, 2048)
    assert device_error_word() == 0 and (np.delete(raw, own, axis=0) == 0x55555555).all()
    x = synth.bf16_bits_to_f32(xb).astype(np.float64)
    check_rows(raw.view(np.float32), host, x[row_of] if gathered else x, counts[:2], offsets[:2], [0, 1])


@pytest.mark.parametrize("f16", [True, False], ids=["f16", "bf16"])
def test_results_scattered_through_y_row_of(st, f16):
    """With y_row_of the results go to rows of the caller's choosing: the same bits as in slot order, and no other row of y is touched."""
    l = ffi.lib()
    dev = MoeLayer.upload(synth.make_layer(39, synth.MoeShape(experts=16)), st)
    counts = np.array([0, 3, 0, 2, 1, 40, 0, 9, 0, 70, 8, 16, 17, 5, 0, 1], dtype=np.int32)
    offsets = (np.cumsum(counts) - counts).astype(np.int32)
    n, rows, rng = int(counts.sum()), int(counts.sum()) + 37, np.random.Generator(np.random.PCG64(9))
    xf = rng.standard_normal((n, 2048), dtype=np.float32)
    xf[::3] *= 0.004  # bf16: rows that are divided by a power of two on the way
    to = rng.permutation(rows)[:n].astype(np.int32)
    dx = DevBuf.from_array(xf.astype(np.float16) if f16 else synth.f32_to_bf16_bits(xf), st)
    dcnt, doff, dto = (DevBuf.from_array(a, st) for a in (counts, offsets, to))
    dact, dsh = DevBuf(n * 1024), DevBuf(16)
    w = (*dev.gate_up.expert(0), *dev.down.expert(0), *dev.shared_gate_up.rows(0), *dev.shared_down.rows(0))
    got = []
    for y_row_of in (NULL, dto.at(0)):
        dy = DevBuf(rows * 8192)
        dy.fill(0x55, st)
        launched(l.drb_moe_prefill_block(*w, dx.at(0), NULL, doff.at(0), dcnt.at(0), dact.at(0), dy.at(0), dact.at(0), dsh.at(0), 0, 16, 2048, 512,
                                         int(f16), y_row_of, st.raw), "block")
        got.append(dy.download(np.uint32, rows * 2048, st).reshape(rows, 2048))
    assert device_error_word() == 0 and np.isfinite(got[0][:n].view(np.float32)).all()
    assert np.array_equal(got[1][to], got[0][:n])
    assert (np.delete(got[1], to, axis=0) == 0x55555555).all() and (got[0][n:] == 0x55555555).all()


@pytest.mark.parametrize("experts,topk", [(256, 8), (64, 32), (32, 32), (40, 1)])
@pytest.mark.parametrize("rows", [1, 7, 32, 33, 150])
def test_layer_call_equals_the_separate_calls(st, experts, topk, rows):
    """drb_moe_prefill_layer against the calls that it stands for, with a logit bias: the same bits in rows, logits, routing and x. top-k up
    to 32, as dr_moe_topk takes it."""
    l = ffi.lib()
    dev = MoeLayer.upload(synth.make_layer(40, synth.MoeShape(experts=experts)), st)
    x = synth.make_x(41, rows, 2048)
    bias = DevBuf.from_array(np.random.Generator(np.random.PCG64(7)).standard_normal((rows, experts + 1), dtype=np.float32), st)
    one, sep = MoePrefill(dev, rows, topk, st=st), MoePrefill(dev, rows, topk, st=st)
    for p in (one, sep):
        p.logit_bias = bias
        p.x.upload(x, st)
    one.run_device(rows)
    sep.route_device(rows)
    launched(l.drb_moe_group(sep.idx.at(0), rows, topk, 0, experts, sep.counts.at(0), sep.offsets.at(0), sep.slot_of.at(0), sep.row_of.at(0), st.raw), "group")
    w = (*dev.gate_up.expert(0), *dev.down.expert(0), *dev.shared_gate_up.rows(0), *dev.shared_down.rows(0))
    launched(l.drb_moe_prefill_block(*w, sep.hn_b.at(0), sep.row_of.at(0), sep.offsets.at(0), sep.counts.at(0), sep.ap.at(0), sep.yp.at(0), sep.sh_act_b.at(0),
                                     sep.sh_out.at(0), rows, experts, 2048, 512, 1, NULL, st.raw), "block")
    launched(l.dr_moe_combine(sep.x.at(0), sep.yp.at(0), sep.slot_of.at(0), sep.wts.at(0), sep.sgate.at(0), sep.sh_out.at(0), rows, topk, 2048, st.raw), "combine")
    for name, count in (("hn_b", rows * 1024), ("rlog", rows * (experts + 1)), ("idx", rows * topk), ("wts", rows * topk), ("sgate", rows),
                        ("counts", experts), ("offsets", experts), ("x", rows * 2048)):
        a, b = (getattr(p, name).download(np.uint32, count, st) for p in (one, sep))
        assert np.array_equal(a, b), name
    assert np.isfinite(one.x.download(np.float32, rows * 2048, st)).all() and device_error_word() == 0


@pytest.mark.parametrize("f16,bar", [(True, 1.0e-7), (False, 8.5e-8)], ids=["f16", "bf16"])
def test_router_logits_keep_the_precision_of_an_fma_chain(st, f16, bar):
    """2-norm of the error against fp64 over 300 normalised rows. The bars: a chain of fp32 FMAs per lane with a butterfly behind it, which
    these logits once were, measures 1.08e-7 (fp16 rows) and 8.0e-8 (bf16 rows); the tree of sums on mma.sync 8.4e-8 and 7.5e-8."""
    rng = np.random.Generator(np.random.PCG64(300))
    x = rng.standard_normal((300, 2048), dtype=np.float32)
    xb = x.astype(np.float16) if f16 else synth.f32_to_bf16_bits(x)
    wb = synth.f32_to_bf16_bits(rng.standard_normal((257, 2048), dtype=np.float32) * 0.02)
    dx, dw, dl = DevBuf.from_array(xb, st), DevBuf.from_array(wb, st), DevBuf(300 * 257 * 4)
    call = ffi.lib().drb_router_logits_f16 if f16 else ffi.lib().drb_router_logits
    launched(call(dx.at(0), dw.at(0), dl.at(0), 300, 257, 2048, 0.0, st.raw), "router_logits")
    ref = (xb.astype(np.float64) if f16 else synth.bf16_bits_to_f32(xb).astype(np.float64)) @ synth.bf16_bits_to_f32(wb).astype(np.float64).T
    err = np.linalg.norm(dl.download(np.float32, 300 * 257, st).reshape(300, 257) - ref) / np.linalg.norm(ref)
    assert err <= bar, err
