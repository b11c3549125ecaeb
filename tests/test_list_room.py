"""Regions of the member lists (rd_listroom.hpp, compiled for the host): whatever the
members' distribution over the keys, the regions that the kernels lay out fit the rows
that the host allocates."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include "rd_listroom.hpp"
#include <cstdio>
int main()
{
    int64_t n = 0, ns = 0, used = 0;
    int k;
    while (scanf("%d", &k) == 1) { n += k; ++ns; used += rdb::list_room(k); if (rdb::list_room(k) <= k) return 2; }
    printf("%lld %lld\n", (long long)used, (long long)rdb::list_rows(n, ns));
}
"""


@pytest.fixture(scope="module")
def room(tmp_path_factory):
    d = tmp_path_factory.mktemp("listroom")
    src, exe = d / "t.cpp", d / "t"
    src.write_text(PROGRAM)
    inc = os.path.join(ROOT, "ridgedetection_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-I", inc, str(src), "-o", str(exe)], check=True)

    def run(counts):
        out = subprocess.run([str(exe)], input=" ".join(map(str, counts)), check=True,
                             capture_output=True, text=True).stdout
        return tuple(map(int, out.split()))
    return run


@pytest.mark.parametrize("seed", range(6))
def test_regions_fit(room, seed):
    r = np.random.default_rng(seed)
    counts = np.concatenate([r.integers(0, 4, 500), r.integers(0, 40_000, 50),
                             [0, 1, 2, 3, 4, 5, 7, 8, 10 ** 9][: 8 + seed % 2]])
    used, rows = room(counts)
    assert used <= rows


def test_sizes_are_stated_once():
    """The host sizes and the kernels' layout come from the same functions."""
    csrc = os.path.join(ROOT, "ridgedetection_b200", "csrc")
    host, dev = (open(os.path.join(csrc, f)).read() for f in ("rd_engine.cu", "rd_kernels.cu"))
    assert "list_rows(" in host and "CAND_MAX * blocks" in host
    assert "list_room(n)" in dev and "at < CAND_MAX" in dev


def test_limits_are_per_cloud(tmp_path):
    src, exe = tmp_path / "l.cpp", tmp_path / "l"
    src.write_text('#include "rd_listroom.hpp"\n#include <cstdio>\n#include <cstdlib>\n'
                   'int main(int, char** a) { printf("%d", rdb::lists_possible(atoll(a[1]), atoll(a[2]))); }\n')
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "ridgedetection_b200", "csrc"), str(src),
                    "-o", str(exe)], check=True)

    def possible(n, ns):
        return subprocess.run([str(exe), str(n), str(ns)], check=True, capture_output=True, text=True).stdout == "1"
    assert possible(10 ** 6, 10 ** 6) and possible(2 ** 30, 1000) and possible(0, 5)
    assert not possible(2 ** 30 + 1, 1)                 # positions of the edits
    assert not possible(2 ** 28, 2 ** 28)               # rows past 2^31
    # the batch has no say: the engine asks for every cloud, and sorts up to 2^31 points
    host = open(os.path.join(ROOT, "ridgedetection_b200", "csrc", "rd_engine.cu")).read()
    assert "lists_possible(cd.n_all, cd.ns_cap)" in host and "total_points <= (int64_t(1) << 30)" not in host
