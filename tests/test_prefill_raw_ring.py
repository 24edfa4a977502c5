"""The ring of raw weight stages in the grouped prefill GEMMs, followed step by step on the CPU with boxes that land in any order.

An mbarrier wait tests one bit of the phase: it takes a use of a stage for landed when the use before it is still in flight. Two
groups of convert warps take turns at the steps, so a stage's previous use may be the other group's. The walk keeps, for the group
of each step, what it knows to have landed: what it has waited for itself, and what the waits for the MMAs of earlier steps imply.
Every wait for a stage has to find the use before it among that. The order of the waits and the ring's sizes are read
from the source."""

from __future__ import annotations

import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "drama_rs_b200", "csrc", "moe_prefill_tc.cuh")


def source() -> str:
    with open(SRC) as f:
        return f.read()


def branches() -> tuple[str, str]:
    """The int4 and the 8-bit half of the convert warps' step loop."""
    s = source()
    body = s[s.index("// ================= convert warps") : s.index("// ================= MMA warp")]
    body = body[body.index("Ring<(NSM ? NSM : 1)> rs;  // int4 items' scales") :]
    return tuple(body.split("} else {  // 8-bit weights"))


def mma_wait_first(branch: str) -> bool:
    return 0 <= branch.find("a_wait();") < branch.index("ctl.rawfull")


def walk(raws: list[int], nraw: int, nst: int, groups: int, first: list[bool]) -> list[int]:
    """raws[s]: raw stages of step s; first[s]: the step waits for its MMA stage ahead of its raw stages. Returns the steps whose wait
    for a raw stage cannot be trusted."""
    start = [sum(raws[:s]) for s in range(len(raws) + 1)]
    step_of = [s for s, n in enumerate(raws) for _ in range(n)]
    waited = [set() for _ in range(groups)]  # raw requests a group has waited for
    implied = [-1] * groups                  # every step up to this one has been converted, as far as the group knows
    bad = []
    for s, n in enumerate(raws):
        g = s % groups
        if first[s]:
            implied[g] = max(implied[g], s - nst)
        for r in range(start[s], start[s] + n):
            before = r - nraw
            if before >= 0 and before not in waited[g] and step_of[before] > implied[g]:
                bad.append(s)
        waited[g].update(range(start[s], start[s] + n))
        implied[g] = max(implied[g], s - nst)
    return bad


ITEMS = ["ssssss", "iiiiii", "ssiii", "sisisi", "siisii", "issi"]  # shared-expert (8-bit) and int4 items of one block, in any order


@pytest.mark.parametrize("items", ITEMS)
@pytest.mark.parametrize("gemm,nraw,nstep", [(0, 5, 8), (1, 6, 2)])
def test_every_raw_wait_is_unambiguous(gemm, nraw, nstep, items):
    s = source()
    assert re.search(r"NRAW = FMT == 1 \? 10 : GEMM == 0 \? 5 : 6;", s) and re.search(r"constexpr int NST = 3;", s)
    assert "GROUPS = FMT == 1 ? 1 : 2" in s
    int4, eight = branches()
    order = {"i": mma_wait_first(int4), "s": mma_wait_first(eight)}
    raws = [2 if it == "s" else 1 for it in items for _ in range(nstep)]
    first = [order[it] for it in items for _ in range(nstep)]
    assert walk(raws, nraw, 3, 2, first) == []


def test_the_walk_sees_the_hazard():
    """With the raw stages waited for first, 8-bit steps run into the other group's boxes, and so do the first int4 steps behind them;
    int4 steps among themselves and a single group do not."""
    assert walk([2] * 16, 5, 3, 2, [False] * 16) and walk([2] * 16, 6, 3, 2, [False] * 16)
    assert walk([2] * 8 + [1] * 8, 6, 3, 2, [True] * 8 + [False] * 8)
    assert walk([1] * 32, 5, 3, 2, [False] * 32) == []
    assert walk([2] * 32, 10, 3, 1, [False] * 32) == []
