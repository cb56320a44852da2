"""Index sums of the row views (row_elements, VecField::covers) stay below 2^31 for
every cell of a grid that they admit. The header's rule is compiled for the host; the
device's sum is restated in Python's integers."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "pic_types.h"
int main(int argc, char** argv) {
  const int ext[3] = { std::atoi(argv[1]), std::atoi(argv[2]), std::atoi(argv[3]) };
  const int64_t s[4] = { std::atoll(argv[4]), std::atoll(argv[5]), std::atoll(argv[6]), std::atoll(argv[7]) };
  std::printf("%d\n", pic::row_elements(reinterpret_cast<const void*>(std::atoll(argv[8])), ext, s, std::atoi(argv[9])));
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("rows")
    src = d / "rows.cpp"
    src.write_text(SRC)
    exe = str(d / "rows")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "entity_gb300", "csrc"), "-o", exe, str(src)])
    return lambda *a: int(subprocess.check_output([exe, *map(str, a)]))


def _covers(ext, s, ng, order):
    """The largest sum of covers<order + 1> over the cells of the grid (the caller adds one to each index)."""
    n = order + 1
    top = [e - 2 * ng - 1 + ng + 1 if e > 1 else 0 for e in ext]
    return top[0] + (top[1] + n) * s[1] + (top[2] + n) * s[2] + 5 * s[3] + n + 8


@pytest.mark.parametrize("n", [8, 96, 256, 600, 700, 703, 704, 705, 706, 707, 800])
@pytest.mark.parametrize("ng", [2])
def test_admitted_grids_stay_below_32_bits(rule, n, ng):
    for ext in ((n + 2 * ng,) * 3, (n + 2 * ng, 2 * n, n // 2 + 2 * ng)):
        s = (1, ext[0], ext[0] * ext[1], ext[0] * ext[1] * ext[2])
        got = rule(*ext, *s, 4096, 6)
        count = 6 * ext[0] * ext[1] * ext[2]
        worst = max(_covers(ext, s, ng, o) for o in (1, 2))
        assert got in (0, count)
        if got:
            assert worst < 2 ** 31
        # and refuses little that would do: four rows and planes
        if count + 5 * (s[1] + s[2]) < 2 ** 31 - 100:
            assert got == count


def test_padded_strides_and_refusals(rule):
    ext, ng = (36, 20, 20), 2
    for s3 in ((2 ** 31 - 20000) // 5, (2 ** 31 - 40000) // 5, (2 ** 31 - 60000) // 5):
        s = (1, 36, 720, s3)
        if rule(*ext, *s, 256, 6):
            assert _covers(ext, s, ng, 2) < 2 ** 31
    assert rule(36, 20, 20, 1, 36, 720, 14400, 256, 6) == 6 * 14400
    assert rule(36, 20, 20, 1, 36, 720, 14400, 260, 6) == 0   # not on 16 bytes
    assert rule(36, 20, 20, 6, 216, 4320, 1, 256, 6) == 0     # components innermost
    assert rule(36, 20, 20, 1, 36, 720, 14400, 0, 6) == 0
