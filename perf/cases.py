"""The work that a host of this library has it do, as timed cases.

A case is a plain dict with a "kind":

  gemv         one int8 GEMV call (`dr_gemv_q8`): a vocabulary head, or any projection issued by itself
  chain        the dense GEMVs of a decode step between the MoE blocks, captured once and replayed: per backbone layer
               an in-projection (RMSNorm fused) and an out-projection (residual fused), per tower layer the attention
               projections and a SwiGLU MLP, at the end a bf16 head; every op prefetches the next one's weights
  decode       a batch-1 step through the per-layer entry points of the ABI (`MoeDecoder`), int4 or block-FP8 experts
  stack        a batch-1 step through the persistent kernel (`MoeStackDecoder`)
  prefill      one MoE block over a chunk of rows through the library's own sequence (`MoePrefill`)
  prefill_abi  the same block with the reference host's call sequence (`MoePrefill(reference_calls=True)`)
  prefill_fp8  the expert GEMMs over block-FP8 experts (`dr_moe_prefill_fp8`) on rows already sorted by expert
  quant        a checkpoint's expert tensor quantised on the device (`drb_quant_q4`, `drb_quant_q8`)

Weights, activations and routing follow the distributions of `drama_rs_b200.synth`, drawn on the GPU from the seed.
The expert-parallel path needs more than one GPU to be what it is and has no case here.
"""

from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from drama_rs_b200 import ffi, synth
from drama_rs_b200.engine import MoeDecoder, MoePrefill, MoeStackDecoder
from drama_rs_b200.gpu import ExtBuf, Graph, Stream, check, launched
from drama_rs_b200.model import Q4, Q8, Fp8Experts, MoeLayer

SHAPE = synth.MoeShape()
H, I, TOPK, EPS = SHAPE.hidden, SHAPE.inter, SHAPE.topk, SHAPE.eps
NULL = C.c_void_p(0)
GEMV_K = (512, 2048, 4096, 6144, 8192)  # the input sizes that dr_gemv_q8 takes
TOWER_I, HEAD_ROWS = 6144, 4097         # a tower layer's MLP width, the bf16 head's rows


def listed() -> list[dict]:
    return [
        # the vocabulary head of the GEMV sweep: one long stream of weights
        {"name": "lm_head", "kind": "gemv", "n": 151936, "k": 2048, "norm": True, "res": False},
        # the projections around the MoE blocks, many short launches one behind the other
        {"name": "gemv_chain", "kind": "chain", "layers": 8, "towers": 4},
        # a host that keeps the reference's two calls per MoE layer
        {"name": "decode_abi", "kind": "decode", "layers": 8, "experts": 256, "fp8": False},
        # the same over the checkpoint's own block-FP8 experts
        {"name": "decode_fp8", "kind": "decode", "layers": 8, "experts": 256, "fp8": True},
        # the whole 40-layer step of the benchmark
        {"name": "decode_stack40", "kind": "stack", "layers": 40, "experts": 256},
        # the tail of a chunked prompt: a handful of rows, launches and latency
        {"name": "prefill_5", "kind": "prefill", "rows": 5, "zipf": 0.0},
        # 64 streams decoding together, one row each, uniform routing
        {"name": "prefill_64", "kind": "prefill", "rows": 64, "zipf": 0.0},
        # the benchmark's prefill: 300 rows, expert popularity after Zipf(1.1)
        {"name": "prefill_300", "kind": "prefill", "rows": 300, "zipf": 1.1},
        # a long prompt's chunk
        {"name": "prefill_2048", "kind": "prefill", "rows": 2048, "zipf": 1.1},
        # 300 rows as the reference's host issues them: cuBLAS, counts to the host, a host scan
        {"name": "prefill_abi_300", "kind": "prefill_abi", "rows": 300, "zipf": 1.1},
        # 300 rows over block-FP8 experts
        {"name": "prefill_fp8_300", "kind": "prefill_fp8", "rows": 300, "zipf": 1.1},
        # a quarter of a layer's gate/up experts on their way from the checkpoint to int4
        {"name": "quant_q4", "kind": "quant", "bits": 4, "experts": 64, "n": 1024, "k": 2048},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(("gemv", "chain", "decode", "stack", "prefill", "prefill", "prefill_abi", "prefill_fp8", "quant"))
    if kind == "gemv":
        k = rng.choice(GEMV_K)
        return {"kind": kind, "n": _log_int(rng, 16, 151936 * 2048 // max(k, 2048)), "k": k, "norm": rng.random() < 0.5, "res": rng.random() < 0.5}
    if kind == "chain":
        return {"kind": kind, "layers": rng.randint(1, 12), "towers": rng.randint(0, 4)}
    if kind == "decode":
        return {"kind": kind, "layers": rng.randint(1, 8), "experts": rng.choice((16, 64, 128, 256)), "fp8": rng.random() < 0.5}
    if kind == "stack":
        return {"kind": kind, "layers": rng.randint(1, 40), "experts": rng.choice((64, 128, 256))}
    if kind == "quant":
        return {"kind": kind, "bits": rng.choice((4, 8)), "experts": rng.randint(1, 64), "n": rng.choice((257, 512, 1001, 1024)),
                "k": rng.choice((512, 2048))}
    return {"kind": kind, "rows": _log_int(rng, 1, 2048), "zipf": rng.choice((0.0, 1.1))}


# ----------------------------------------------------------------------------- inputs

_STREAM: Stream | None = None


def _stream() -> Stream:
    """The one stream that a host keeps for its launches."""
    global _STREAM
    if _STREAM is None:
        _STREAM = Stream()
    return _STREAM


def _ext(t: torch.Tensor) -> ExtBuf:
    return ExtBuf(t.data_ptr(), t.numel() * t.element_size(), keep=t)


def _p(t: torch.Tensor) -> C.c_void_p:
    return C.c_void_p(t.data_ptr())


class _Draw:
    """Seeded device tensors in the converter's layouts."""

    def __init__(self, seed: int) -> None:
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def randn(self, *shape: int) -> torch.Tensor:
        return torch.randn(shape, device="cuda", generator=self.g)

    def q8(self, n: int, k: int) -> tuple[torch.Tensor, torch.Tensor]:
        q = torch.randint(-127, 128, (n, k), dtype=torch.int8, device="cuda", generator=self.g)
        row = (self.randn(n, 1) * 0.005).abs().clamp_min(1e-4).half()
        return q, row.expand(n, k // 128).contiguous()

    def q8_weight(self, n: int, k: int) -> Q8:
        q, s = self.q8(n, k)
        return Q8(_ext(q), _ext(s), n, k)

    def q4(self, e: int, n: int, k: int) -> Q4:
        q = torch.randint(0, 256, (e, n, k // 2), dtype=torch.uint8, device="cuda", generator=self.g)
        s = (self.randn(e, n, k // 64) * 0.01).abs().clamp_min(1e-4).half()
        sm = torch.stack((s, (s.float() * -8.0).half()), dim=-1).contiguous()
        return Q4(_ext(q), _ext(sm), e, n, k)

    def fp8(self, e: int, n: int, k: int) -> tuple[torch.Tensor, torch.Tensor]:
        w = torch.empty((e, n, k), dtype=torch.uint8, device="cuda")
        for lo in range(0, e, 32):
            part = (self.randn(min(32, e - lo), n, k) * 112.0).clamp_(-448.0, 448.0)
            w[lo : lo + 32] = part.to(torch.float8_e4m3fn).view(torch.uint8)
        return w, (self.randn(e, n // 128, k // 128).abs() * (0.01 / 112.0)).clamp_min(1e-7)

    def fp8_experts(self, e: int) -> Fp8Experts:
        gw, gs = self.fp8(e, 2 * I, H)
        dw, ds = self.fp8(e, H, I)
        return Fp8Experts(_ext(gw), _ext(gs), _ext(dw), _ext(ds), e, H, I)

    def layer(self, e: int, int4: bool = True) -> MoeLayer:
        """One MoE layer; without int4 experts (a block-FP8 model has none) the int4 tensors hold one expert."""
        router = (self.randn(e + 1, H) * 0.02).bfloat16()
        norm = 1.0 + self.randn(H) * 0.1
        held = e if int4 else 1
        return MoeLayer(_ext(router), _ext(norm), self.q8_weight(2 * I, H), self.q8_weight(H, I), self.q4(held, 2 * I, H), self.q4(held, H, I), e, H, I)

    def rows(self, n: int) -> torch.Tensor:
        return self.randn(n, H).bfloat16().float()


def _bias(seed: int, zipf: float) -> np.ndarray | None:
    return synth.zipf_router_bias(seed, SHAPE.experts, zipf) if zipf else None


def prepare(case: dict, seed: int):
    st, d = _stream(), _Draw(seed)
    state = {"kind": case["kind"]}
    if case["kind"] == "gemv":
        n, k = case["n"], case["k"]
        w, s = d.q8(n, k)
        state.update(w=w, s=s, x=d.randn(k).bfloat16().float(), y=torch.empty(n, device="cuda"), n=n, k=k,
                     nw=1.0 + d.randn(k) * 0.1 if case["norm"] else None, res=d.randn(n) if case["res"] else None)
    elif case["kind"] == "chain":
        state.update(_chain(d, case["layers"], case["towers"], st))
    elif case["kind"] == "decode":
        layers = [d.layer(case["experts"], not case["fp8"]) for _ in range(case["layers"])]
        fp8 = [d.fp8_experts(case["experts"]) for _ in layers] if case["fp8"] else None
        state.update(dec=MoeDecoder(layers, TOPK, EPS, st, fp8=fp8), x=d.rows(1)[0].cpu().numpy())
        torch.cuda.synchronize()
        state["dec"].capture()
    elif case["kind"] == "stack":
        layers = [d.layer(case["experts"]) for _ in range(case["layers"])]
        torch.cuda.synchronize()
        state.update(dec=MoeStackDecoder(layers, TOPK, EPS, st), x=d.rows(1)[0].cpu().numpy())
        state["dec"].capture()
    elif case["kind"] in ("prefill", "prefill_abi"):
        n = case["rows"]
        pre = MoePrefill(d.layer(SHAPE.experts), n, TOPK, EPS, st, reference_calls=case["kind"] == "prefill_abi")
        x, out = d.rows(n), torch.empty((n, H), device="cuda")
        pre.x = _ext(out)
        bias = _bias(seed, case["zipf"])
        if bias is not None:
            rows = torch.zeros((n, SHAPE.experts + 1), device="cuda")
            rows[:, : SHAPE.experts] = torch.from_numpy(bias).cuda()
            pre.logit_bias = _ext(rows)
        state.update(pre=pre, x=x, out=out, n=n)
    elif case["kind"] == "prefill_fp8":
        n, e = case["rows"], SHAPE.experts
        logits = d.randn(n, e) * 0.9
        bias = _bias(seed, case["zipf"])
        if bias is not None:
            logits += torch.from_numpy(bias).cuda()
        counts = torch.bincount(logits.topk(TOPK, dim=1).indices.reshape(-1), minlength=e).int()
        state.update(f8=d.fp8_experts(e), counts=counts, offsets=(counts.cumsum(0) - counts).int(), xp=d.randn(n * TOPK, H).bfloat16(),
                     act=torch.empty((n * TOPK, I), dtype=torch.bfloat16, device="cuda"), y=torch.empty((n * TOPK, H), device="cuda"))
    else:
        group = 64 if case["bits"] == 4 else 128
        w = (d.randn(case["experts"], case["n"], case["k"]) * 0.02).bfloat16().float()  # a bf16 checkpoint widened to f32
        groups = w.numel() // group
        codes = torch.empty((groups, 32), dtype=torch.uint8, device="cuda") if group == 64 else torch.empty((groups, 128), dtype=torch.int8, device="cuda")
        state.update(w=w, groups=groups, bits=case["bits"], q=codes,
                     s=torch.empty((groups, 2) if group == 64 else (groups,), dtype=torch.float16, device="cuda"))
    torch.cuda.synchronize()
    return state


def _chain(d: _Draw, layers: int, towers: int, st: Stream) -> dict:
    """The GEMVs of a decode step in call order, each handed the next one's weights to prefetch (the last one wraps),
    captured into one graph that starts from x0."""
    l = ffi.lib()
    x0, x = d.rows(1)[0], torch.empty(H, device="cuda")
    wide, mid, logits = torch.empty(8192, device="cuda"), torch.empty(TOWER_I, device="cuda"), torch.empty(HEAD_ROWS, device="cuda")
    ops, keep = [], [x0, wide, mid]

    def norm() -> torch.Tensor:
        keep.append(1.0 + d.randn(H) * 0.1)
        return keep[-1]

    def q8(n: int, k: int, src: torch.Tensor, dst: torch.Tensor, nw=None, res=None) -> None:
        w, s = d.q8(n, k)
        keep.extend((w, s))
        ops.append((w, lambda pf, pfb: l.dr_gemv_q8(_p(w), _p(s), _p(src), _p(res) if res is not None else NULL, _p(dst), n, k,
                                                    _p(nw) if nw is not None else NULL, EPS, pf, pfb, st.raw)))

    def swiglu(i: int, src: torch.Tensor, dst: torch.Tensor, nw: torch.Tensor) -> None:
        w, s = d.q8(2 * i, H)
        keep.extend((w, s))
        ops.append((w, lambda pf, pfb: l.dr_gemv_q8_swiglu(_p(w), _p(s), _p(src), _p(dst), i, H, _p(nw), EPS, pf, pfb, st.raw)))

    for _ in range(layers):
        q8(8192, H, x, wide, nw=norm())
        q8(H, 4096, wide, x, res=x)
    for _ in range(towers):
        q8(4096, H, x, wide, nw=norm())
        q8(H, 4096, wide, x, res=x)
        swiglu(TOWER_I, x, mid, norm())
        q8(H, TOWER_I, mid, x, res=x)
    head, head_norm = (d.randn(HEAD_ROWS, H) * 0.02).bfloat16(), norm()
    keep.append(head)
    ops.append((head, lambda pf, pfb: l.dr_gemv_bf16(_p(head), _p(x), _p(logits), HEAD_ROWS, H, _p(head_norm), EPS, pf, pfb, st.raw)))
    torch.cuda.synchronize()

    def record() -> None:
        check(l.dr_d2d(_p(x), _p(x0), H * 4, st.raw), "d2d")
        for i, (_, op) in enumerate(ops):
            nxt = ops[(i + 1) % len(ops)][0]
            launched(op(_p(nxt), nxt.numel() * nxt.element_size()), "gemv")

    return {"graph": Graph(st, record), "keep": keep, "x": x, "logits": logits}


# ----------------------------------------------------------------------------- one pass


def run(state):
    l, st, kind = ffi.lib(), _stream(), state["kind"]
    if kind == "gemv":
        nw, res = state["nw"], state["res"]
        launched(l.dr_gemv_q8(_p(state["w"]), _p(state["s"]), _p(state["x"]), _p(res) if res is not None else NULL, _p(state["y"]), state["n"],
                              state["k"], _p(nw) if nw is not None else NULL, EPS, NULL, 0, st.raw), "gemv_q8")
        return state["y"]
    if kind == "chain":
        state["graph"].launch(st)
        return {"x": state["x"], "logits": state["logits"]}
    if kind in ("decode", "stack"):
        # a token's hidden state in, the new one out, both on the host as the decoders' public calls have them
        state["dec"].set_x(state["x"])
        return state["dec"].step()
    if kind in ("prefill", "prefill_abi"):
        # the block works in place on the rows, which the layer before it has left on the device
        pre = state["pre"]
        check(l.dr_d2d(pre.x.at(0), _p(state["x"]), state["n"] * H * 4, st.raw), "d2d")
        pre.run_device(state["n"])
        return state["out"]
    if kind == "prefill_fp8":
        f8 = state["f8"]
        launched(l.dr_moe_prefill_fp8(f8.gu_w.at(0), f8.gu_s.at(0), f8.d_w.at(0), f8.d_s.at(0), _p(state["xp"]), _p(state["offsets"]),
                                      _p(state["counts"]), _p(state["act"]), _p(state["y"]), f8.e, H, I, st.raw), "moe_prefill_fp8")
        return state["y"]
    quant = l.drb_quant_q4 if state["bits"] == 4 else l.drb_quant_q8
    launched(quant(_p(state["w"]), state["groups"], _p(state["q"]), _p(state["s"]), st.raw), "quant")
    return {"q": state["q"], "s": state["s"]}


# ----------------------------------------------------------------------------- what a pass cannot do without


def _experts_hit(rows: int, zipf: float) -> int:
    """Experts that the rows reach, from one sample of logits with the spread of the synthetic router."""
    r = np.random.Generator(np.random.PCG64(1))
    logits = r.standard_normal((rows, SHAPE.experts), dtype=np.float32) * np.float32(0.9)
    bias = _bias(1, zipf)
    if bias is not None:
        logits += bias
    return len(np.unique(np.argpartition(-logits, TOPK, axis=1)[:, :TOPK]))


def _q8_bytes(n: int, k: int) -> int:
    return n * k + n * (k // 128) * 2


def work(case: dict) -> dict:
    kind = case["kind"]
    fp8_expert = 3 * H * I + 4 * ((2 * I // 128) * (H // 128) + (H // 128) * (I // 128))
    if kind == "gemv":
        n, k = case["n"], case["k"]
        return {"bytes": _q8_bytes(n, k) + 4 * (k + n) + 4 * k * case["norm"] + 4 * n * case["res"], "flops": 2.0 * n * k}
    if kind == "chain":
        shapes = [(8192, H), (H, 4096)] * case["layers"] + [(4096, H), (H, 4096), (2 * TOWER_I, H), (H, TOWER_I)] * case["towers"]
        return {"bytes": sum(_q8_bytes(n, k) for n, k in shapes) + HEAD_ROWS * (2 * H + 4) + 12 * H,
                "flops": 2.0 * (sum(n * k for n, k in shapes) + HEAD_ROWS * H)}
    if kind in ("decode", "stack"):
        expert = fp8_expert if case.get("fp8") else SHAPE.expert_bytes
        layer = (case["experts"] + 1) * H * 2 + TOPK * expert + SHAPE.shared_bytes + 4 * H
        return {"bytes": case["layers"] * layer + 8 * H, "flops": 2.0 * case["layers"] * ((case["experts"] + 1) * H + (TOPK + 1) * 3 * H * I)}
    if kind in ("prefill", "prefill_abi"):
        n = case["rows"]
        return {"bytes": _experts_hit(n, case["zipf"]) * SHAPE.expert_bytes + SHAPE.shared_bytes + SHAPE.router_bytes + 8 * n * H,
                "flops": 2.0 * n * ((SHAPE.experts + 1) * H + (TOPK + 1) * 3 * H * I)}
    if kind == "prefill_fp8":
        n = case["rows"]
        return {"bytes": _experts_hit(n, case["zipf"]) * fp8_expert + n * TOPK * H * 6, "flops": 2.0 * n * TOPK * 3 * H * I}
    values = case["experts"] * case["n"] * case["k"]
    # int4: 24 clipping candidates, each a quantise, a reconstruction and a squared error
    return {"bytes": values * (4 + 0.5 + 4 / 64 if case["bits"] == 4 else 5 + 2 / 128), "flops": values * (24.0 * 8 if case["bits"] == 4 else 3.0)}


def tolerance(case: dict):
    if case["kind"] == "quant":
        return "exact"  # codes and scales are the converter's, bit for bit
    if case["kind"] in ("gemv", "chain"):
        return {"rel": 2e-5}  # f32 sums over activations of 21 bits; a chain adds its ops' roundings up
    if case["kind"] in ("decode", "stack"):
        return {"rel": 1e-4}  # the same, through up to 40 layers
    # fp16 rows and intermediates (own sequence, FP8 experts); bf16 rows in the reference's sequence
    return {"rel": 5e-3 if case["kind"] == "prefill_abi" else 2e-3}
