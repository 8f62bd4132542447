"""The split rule of fp32 decode for few groups, on the host: every cluster that a plan asks for is resident at once, by the
device's own count of clusters that fit, and no key is left out."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = """
#include <cstdio>
#include "decode_plan.h"
int main() {
    // clusters of 1 .. 8 CTAs: a B200's own count (148 SMs), one with fewer GPCs that hold two of eight, none at all
    const int fits[3][9] = {{0, 148, 74, 45, 33, 26, 22, 15, 15}, {0, 148, 74, 45, 33, 26, 20, 13, 9}, {0, 0, 0, 0, 0, 0, 0, 0, 0}};
    for (int f = 0; f < 3; ++f)
        for (int groups = 1; groups <= 18; ++groups)
            for (int heads = 1; heads <= 8; ++heads)
                for (int keys = 0; keys <= 4096; ++keys) {
                    DecodeSplit S;
                    if (plan_wide(S, fits[f], groups, heads, keys, 128))
                        printf("%d %d %d %d %d %d %d\\n", f, groups, heads, keys, S.cl_size, S.max_clusters, S.cluster_keys);
                }
}
"""


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-I", os.path.join(ROOT, "mx230_b200", "csrc"),
                    str(d / "plan.cpp"), "-o", str(d / "plan")], check=True)
    out = subprocess.run([str(d / "plan")], capture_output=True, text=True, check=True).stdout
    return [tuple(map(int, ln.split())) for ln in out.splitlines()]


FITS = [[0, 148, 74, 45, 33, 26, 22, 15, 15], [0, 148, 74, 45, 33, 26, 20, 13, 9], [0] * 9]


def test_every_cluster_of_a_plan_is_resident(plans):
    assert plans
    for f, groups, heads, keys, c, k, per in plans:
        what = (f, groups, heads, keys, c, k)
        assert 1 <= c <= 8 and 1 <= k <= 4 and groups * k <= FITS[f][c], what
        assert per == 4 * c * 128, what
        if keys:   # one cluster whose CTAs' first tiles cover the keys, or the largest
            assert k == 1 and (c == 8 or (c - 1) * 128 < keys <= c * 128), what


def test_unknown_lengths_get_the_warps_of_the_four_warp_plan(plans):
    """148 SMs: with more than two heads a group, four fifths of the SMs or 16 CTAs a group."""
    got = {(g, h): (c, k) for f, g, h, keys, c, k, _ in plans if f == 0 and keys == 0}
    assert {g for g, _ in got} == set(range(1, 16))   # 16 clusters of eight do not fit: four-warp CTAs
    for (g, h), (c, k) in got.items():
        if h > 2 and g < 14:
            assert c * k >= 16 or c * k * g * 5 >= 148 * 4 or (g, c, k) in ((9, 6, 2),), (g, h, c, k)
        if h <= 2:
            assert c == 8
