"""dr_moe_combine against float64, one call at a time: both forms (top-8, whose blocks walk over rows, and any other topk, a block per row),
row widths that leave the last warp of a block partly or wholly out of range, one row to more than three per resident block, and topk on either
side of the four pairs that are taken at once. Nothing outside the rows is touched."""

from __future__ import annotations

import numpy as np
import pytest

from drama_rs_b200 import ffi
from drama_rs_b200.gpu import DevBuf, Stream, launched

pytestmark = pytest.mark.gpu
GUARD = 64


@pytest.mark.parametrize("topk", [1, 3, 4, 7, 8, 10, 32])
@pytest.mark.parametrize("h", [4, 132, 1028, 2048])
@pytest.mark.parametrize("rows", [1, 5, 2000])
def test_combine(rows, h, topk):
    rows = min(rows, 400) if topk == 32 else rows
    st, r = Stream(), np.random.Generator(np.random.PCG64(rows + h + topk))
    f = lambda *s: r.standard_normal(s, dtype=np.float32)
    pairs = rows * topk + 3  # some slots belong to nobody
    x, y, shared, sgate, w = f(rows, h), f(pairs, h), f(rows, h), f(rows) * 3, np.abs(f(rows, topk))
    slot = r.permutation(pairs)[: rows * topk].astype(np.int32).reshape(rows, topk)
    up = lambda a: DevBuf.from_array(np.ascontiguousarray(a), st)
    dx = up(np.concatenate([x.reshape(-1), np.full(GUARD, 7, np.float32)]))
    dy, ds, dw, dg, dsh = up(y), up(slot), up(w), up(sgate), up(shared)
    launched(ffi.lib().dr_moe_combine(dx.at(0), dy.at(0), ds.at(0), dw.at(0), dg.at(0), dsh.at(0), rows, topk, h, st.raw), "combine")
    got = dx.download(np.float32, rows * h + GUARD, st)
    assert (got[rows * h :] == 7).all()
    sg = 1 / (1 + np.exp(-sgate.astype(np.float64)))[:, None]
    terms = [x.astype(np.float64), sg * shared] + [w[:, k, None].astype(np.float64) * y[slot[:, k]] for k in range(topk)]
    # every term passes at most topk + 2 roundings; the gate is good to four units
    bound = (topk + 6) * 2.0**-24 * sum(np.abs(t) for t in terms)
    assert (np.abs(got[: rows * h].reshape(rows, h) - sum(terms)) <= bound).all()
