"""What the GEMVs ask for on a caller's prefetch hint: the kernel's own function, compiled for the host with a prefetch that records."""

from __future__ import annotations

import os
import shutil
import subprocess

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "drama_rs_b200", "csrc", "gemv.cuh")
SKIP, SMS = 96 * 1024, 148

MAIN = r"""
#include <cstddef>
#include <cstdio>
#include <cstdlib>
#define DRB_DEV static
static const char* base = (const char*)4096;
// the share of [pf, pf + bytes) that one block of `blocks` prefetches, as csrc/common.cuh cuts it (pieces begin and end on 16 bytes)
static void prefetch_share(const char* pf, size_t bytes, unsigned block, unsigned blocks) {
  if (!pf || bytes == 0) return;
  const size_t lo = ((size_t)pf + 15) & ~(size_t)15, hi = ((size_t)pf + bytes) & ~(size_t)15;
  if (hi <= lo) return;
  const size_t per = (((hi - lo + blocks - 1) / blocks) + 15) & ~(size_t)15, b0 = block * per, b1 = b0 + per < hi - lo ? b0 + per : hi - lo;
  if (b0 < b1) printf("%zu %zu\n", lo + b0 - (size_t)base, b1 - b0);
}
@HINT@
int main(int, char** v) {
  const size_t bytes = strtoull(v[1], 0, 10);
  const unsigned skip = atoi(v[2]), blocks = atoi(v[3]);
  for (unsigned b = 0; b < blocks; ++b) prefetch_hint(base, bytes, skip, @SMS@ b, blocks);
}
"""


@pytest.fixture(scope="module")
def hint(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    with open(SRC) as f:
        s = f.read()
    start = s.index("constexpr size_t HINT_WHOLE") if "HINT_WHOLE" in s else s.index("DRB_DEV void prefetch_hint")
    code = s[start : s.index("constexpr unsigned HINT_SKIP")]
    d = tmp_path_factory.mktemp("hint")
    (d / "hint.cpp").write_text(MAIN.replace("@HINT@", code).replace("@SMS@", f"{SMS}u," if "unsigned sms" in code else ""))
    subprocess.run(["g++", "-std=c++17", "-o", str(d / "hint"), str(d / "hint.cpp")], check=True)

    def covered(region: int, skip: int, blocks: int) -> np.ndarray:
        out = subprocess.run([str(d / "hint"), str(region), str(skip), str(blocks)], capture_output=True, text=True, check=True).stdout
        got = np.zeros(region // 16 + 1, dtype=np.int32)
        for line in out.splitlines():
            at, n = map(int, line.split())
            assert at % 16 == 0 and n % 16 == 0 and at + n <= region
            got[at // 16 : (at + n) // 16] += 1
        return got[: region // 16]

    return covered


@pytest.mark.parametrize("blocks", [1, 17, SMS])
@pytest.mark.parametrize("region", [257 * 4096, 2 << 20, 48])
def test_small_regions_are_prefetched_whole(hint, region, blocks):
    assert (hint(region, SKIP, blocks) == 1).all()


@pytest.mark.parametrize("blocks", [1, 40, 147, SMS])
@pytest.mark.parametrize("region", [8192 * 2048, 12288 * 2048, 4097 * 4096])
def test_large_regions_leave_out_what_the_successor_requests_itself(hint, region, blocks):
    got = hint(region, SKIP, blocks)
    share = region // SMS
    want = np.zeros_like(got)
    for i in range(SMS):
        want[-(-(i * share + SKIP) // 16) : (i * share + min(share, SKIP + 131072)) // 16] = 1
    assert np.array_equal(got, want)


def test_without_overlap_the_whole_region(hint):
    assert (hint(8192 * 2048, 0, SMS) == 1).all()
