"""Neighbour lists of a decimation whose lengths add up to more than 32 bits hold:
46,342 points that all lie within 2 r2 of one another have 2^31 list entries.  The
rule the kernels ask (rd_listfit.hpp) runs here on the CPU; a total taken in 32 bits
is negative there, passes for small, and the lists are written far out of range."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ridgedetection_b200", "csrc")

PROGRAM = r"""
#include "rd_listfit.hpp"
#include <cstdio>
#include <cstdlib>
int main(int, char** a)
{
    const int64_t n = atoll(a[1]), len = atoll(a[2]), room = atoll(a[3]);
    int64_t total = 0;
    for (int64_t i = 0; i < n; ++i) total += rdb::list_len((int)len);
    // what one warp of the scan adds in 32 bits
    if (32ll * rdb::list_len((int)len) > INT32_MAX) return 2;
    printf("%d\n", rdb::lists_fit(total, room) ? 1 : 0);
    return 0;
}
"""


@pytest.fixture(scope="module")
def fits(tmp_path_factory):
    d = tmp_path_factory.mktemp("listfit")
    src, exe = d / "t.cpp", d / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)

    def run(n, length, room):
        out = subprocess.run([str(exe), str(n), str(length), str(room)], check=True,
                             capture_output=True, text=True).stdout
        return out.strip() == "1"
    return run


@pytest.mark.parametrize("n,length,room,want", [
    (5_000, 40, 5_000 * 4_096, True),
    (10_000, 4_096, 10_000 * 4_096, True),
    (10_000, 4_097, 10_000 * 4_096, False),
    (46_341, 46_340, 46_341 * 4_096, False),      # just below 2^31 entries
    (46_342, 46_341, 46_342 * 4_096, False),      # 2^31 and more
    (65_537, 65_536, 65_537 * 4_096, False),      # 2^32 + 65,536: wraps to 65,536
    (80_000_000, 30, 80_000_000 * 32, False),     # fits the room, not the offsets
    (70_000_000, 70_000_000, 70_000_000 * 32, False),
])
def test_lists_fit(fits, n, length, room, want):
    assert fits(n, length, room) is want


def test_scans_use_the_rule():
    """Both scans of list lengths (one CTA's and the GPU-wide one) add in 64 bits."""
    for f in ("rd_grid.cuh", "rd_kernels.cu"):
        src = open(os.path.join(CSRC, f)).read()
        assert "list_len(nb_off[i])" in src and "lists_fit(" in src, f
        assert "(int64_t)s_carry > " not in src, f
