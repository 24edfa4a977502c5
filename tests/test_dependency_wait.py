"""Programmatic dependent launch: what a kernel may read ahead of its dependency wait. The GEMVs stream their weight matrix early, by
contract; norm and router weights may be the work of the launch before (a host that folds or converts them on the device), so they are
read behind the wait. Read from the source: a stale line would show on the GPU once in a great many runs."""

from __future__ import annotations

import os

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "drama_rs_b200", "csrc")


def ahead_of_the_wait(file: str, namespace: str, kernel: str) -> str:
    with open(os.path.join(CSRC, file)) as f:
        s = f.read()
    s = s[s.index(f"namespace {namespace} {{") :]
    s = s[s.index(f"    {kernel}(") :]
    return s[s.index(") {\n") : s.index("  pdl_wait();")]


@pytest.mark.parametrize("file,namespace,kernel", [("gemv.cuh", "q8", "k_gemv"), ("gemv.cuh", "bf16", "k_gemv"), ("moe_prefill.cuh", "pf", "k_router_logits")])
def test_norm_and_router_weights_are_read_behind_the_wait(file, namespace, kernel):
    body = ahead_of_the_wait(file, namespace, kernel)
    loads = [line for line in body.splitlines() if "__ld" in line and ("(nw" in line or "*>(nw" in line)]
    assert not loads, loads
    if kernel == "k_router_logits":
        calls = body[body.index("auto fetch") :]
        assert "fetch(" not in calls[calls.index("};") :]


@pytest.mark.parametrize("file,kernel", [("moe_decode.cuh", "k_moe_gate_up"), ("moe_decode_fp8.cuh", "k_moe_gate_up_fp8"), ("router.cuh", "k_router_cluster")])
def test_decode_reads_norm_weights_behind_the_wait(file, kernel):
    with open(os.path.join(CSRC, file)) as f:
        s = f.read()
    s = s[s.index(f"    {kernel}(") :]
    s = s[s.index(") {\n") :]
    at = s.find("- consumers\n")  # their own wait: the producer warp has another
    s = s[max(at, 0) :]
    body = s[: s.index("  pdl_wait();")]
    assert not [line for line in body.splitlines() if "(nw)[" in line or "(nw +" in line and "prefetch" not in line]
    assert "(nw)" in s  # the read is where this looks for it
