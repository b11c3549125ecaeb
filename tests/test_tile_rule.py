"""Thresholds of the tiled runs' cluster path (rd_tile_rule.hpp, host code, no GPU
needed): a caller's value holds as given, also one that equals what is reported for
a threshold left to the rule; 0 leaves it to the rule."""
import os
import subprocess

import pytest

import ridgedetection_b200 as rdb

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include "rd_tile_rule.hpp"
#include <cstdio>
#include <cstdlib>
int main(int, char** a)
{
    rdb::TileClusterParams p{atoi(a[1]) != 0, atoi(a[2]), atoi(a[3])};
    const rdb::TileRule r = rdb::tile_rule(p, atoll(a[4]), 148, atoll(a[5]));
    printf("%lld %d %d %d\n", (long long)r.heavy, r.seg_min, (int)r.clusters, (int)r.hand_over);
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("tile_rule")
    src, exe = d / "t.cpp", d / "t"
    src.write_text(PROGRAM)
    inc = os.path.join(ROOT, "ridgedetection_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-I", inc, str(src), "-o", str(exe)], check=True)

    def run(*args):
        out = subprocess.run([str(exe)] + [str(int(x)) for x in args], check=True,
                             capture_output=True, text=True).stdout
        heavy, seg, clusters, hand = out.split()
        return int(heavy), int(seg), clusters == "1", hand == "1"
    return run


@pytest.mark.parametrize("args,want", [
    # enabled, min_points, seg_min, evolve points, largest tile
    ((1, 0, 0, 1_000_000, 50_000), (4096, 12288, True, True)),
    ((1, 0, 0, 10_000_000, 200_000), (16891, 12288, True, True)),
    ((1, 0, 0, 10 ** 9, 200_000), (100000, 12288, True, True)),
    ((1, 0, 0, 1_000_000, 4095), (4096, 12288, False, False)),
    ((1, 100_000, 8192, 1_000_000, 50_000), (100000, 8192, False, False)),
    ((1, 100_000, 8192, 1_000_000, 100_000), (100000, 8192, True, False)),
    ((1, 0, 8192, 1_000_000, 50_000), (4096, 8192, True, True)),
    ((1, 2 ** 31 - 1, 0, 10 ** 9, 10 ** 8), (2 ** 31 - 1, 12288, False, False)),
    ((1, 64, 1, 1_000_000, 100), (64, 1, True, False)),
])
def test_rule(rule, args, want):
    assert rule(*args) == want


def test_off_is_off(rule):
    assert rule(0, 0, 0, 10 ** 7, 10 ** 6)[2:] == (False, False)
    assert rule(0, 64, 1, 10 ** 7, 10 ** 6)[2:] == (False, False)


def test_given_values_are_reported():
    try:
        for m, s in ((100_000, 8192), (99_999, 8193), (1, 1)):
            rdb.set_tile_clusters(True, m, s)
            assert rdb.get_tile_clusters() == (True, m, s)
    finally:
        rdb.set_tile_clusters(True, 0, 0)
