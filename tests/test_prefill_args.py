"""What MoePrefill hands to the one-call prefill: the addresses its weights and buffers have at the time of the call."""

from __future__ import annotations

import ctypes as C
from types import SimpleNamespace

from drama_rs_b200 import ffi
from drama_rs_b200.engine import MoePrefill
from drama_rs_b200.model import Q4, Q8, MoeLayer


class FakeBuf:
    made = 0

    def __init__(self) -> None:
        FakeBuf.made += 1
        self.ptr = 0x1000 * FakeBuf.made


class FakeLib:
    def drb_moe_prefill_layer(self, w, b, *rest) -> int:
        self.w = {n: getattr(w._obj, n) for n, _ in ffi.MoeLayerPtrs._fields_}
        self.b = {n: getattr(b._obj, n) for n, _ in ffi.PrefillBuffers._fields_}
        self.rest = rest
        return 0


def prefill(monkeypatch) -> MoePrefill:
    monkeypatch.setattr("drama_rs_b200.engine.launched", lambda code, what, debug=True: None)
    b = FakeBuf
    layer = MoeLayer(b(), b(), Q8(b(), b(), 1024, 2048), Q8(b(), b(), 2048, 512), Q4(b(), b(), 64, 1024, 2048), Q4(b(), b(), 64, 2048, 512), 64, 2048, 512)
    p = MoePrefill.__new__(MoePrefill)
    p.l, p.st, p.layer, p.topk, p.eps, p.reference_calls, p.rows_f16, p.logit_bias = FakeLib(), SimpleNamespace(raw=None), layer, 8, 1e-6, False, True, None
    for name in ("x", "hn_b", "rlog", "idx", "wts", "sgate", "counts", "offsets", "slot_of", "row_of", "ap", "yp", "sh_act_b", "sh_out"):
        setattr(p, name, b())
    return p


def test_replaced_tensors_are_seen_by_the_next_call(monkeypatch):
    p = prefill(monkeypatch)
    p.run_device(3)
    assert p.l.rest[:5] == (3, 64, 8, 2048, 512)
    first = dict(p.l.w)
    p.layer.down.q, p.layer.router = FakeBuf(), FakeBuf()  # the layer object stays the same
    p.layer.gate_up = Q4(FakeBuf(), FakeBuf(), 64, 1024, 2048)
    p.run_device(3)
    assert p.l.w["d_q"] == p.layer.down.q.ptr != first["d_q"] and p.l.w["router"] == p.layer.router.ptr
    assert p.l.w["gu_q"] == p.layer.gate_up.q.ptr and p.l.w["gu_sm"] == p.layer.gate_up.sm.ptr
    assert p.l.w["sgu_q"] == first["sgu_q"] == p.layer.shared_gate_up.q.ptr
    p.yp.ptr += 64  # another address behind the same object
    p.run_device(3)
    assert p.l.b["y"] == p.yp.ptr
    p.x, p.logit_bias = FakeBuf(), FakeBuf()
    p.run_device(3)
    assert p.l.b["x"] == p.x.ptr and p.l.b["logit_bias"] == p.logit_bias.ptr


def test_the_layer_call_refuses_missing_and_misaligned_buffers():
    """Refused on the host, before the device is looked at."""
    w, b = ffi.MoeLayerPtrs(*range(16, 176, 16)), ffi.PrefillBuffers(*range(16, 256, 16))
    call = lambda: ffi.lib().drb_moe_prefill_layer(C.byref(w), C.byref(b), 4, 16, 8, 2048, 512, 1e-6, None)  # noqa: E731
    vectors = ("x", "rows16", "y", "sh_out", "act", "sh_act", "router", "gu_q", "gu_sm", "d_q", "d_sm", "sgu_q", "sd_q")
    for struct in (w, b):
        for name, _ in struct._fields_:
            p = getattr(struct, name)
            if name != "logit_bias":
                setattr(struct, name, None)
                assert call() == -1, name
            if name in vectors:
                setattr(struct, name, p + 8)
                assert call() == -3, name
            setattr(struct, name, p)
