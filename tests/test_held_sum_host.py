"""The held sums of the raster's tile lists (csrc/held_sum.h), compiled with the
host C++ compiler: exact below the ceiling, the ceiling above it, whatever the
order of the terms -- as the scan over the tiles combines them."""
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "integer_delauney_b200", "csrc")

SOURCE = r"""
#include "held_sum.h"
#include <cstdio>
#include <vector>
int main()
{
    int n;
    while (std::scanf("%d", &n) == 1) {
        std::vector<int32_t> v(n);
        for (auto& x : v) std::scanf("%d", &x);
        int32_t left = 0;
        for (int32_t x : v) left = idl::held_sum(left, x);
        while (v.size() > 1) {   // pairwise, as the shuffles do
            std::vector<int32_t> w;
            for (size_t i = 0; i < v.size(); i += 2) w.push_back(i + 1 < v.size() ? idl::held_sum(v[i], v[i + 1]) : v[i]);
            v = w;
        }
        std::printf("%d %d\n", left, v[0]);
    }
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
def test_sums_stop_at_the_ceiling(tmp_path):
    src, exe = tmp_path / "t.cpp", str(tmp_path / "t")
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", exe], check=True)
    top = 2 ** 31 - 1
    rng = np.random.default_rng(1)
    cases = [[0], [top], [top, 1], [top, top], [2 ** 30] * 5, [2 ** 20] * 4096, [3 << 20] * 2048,
             rng.integers(0, 1000, 8192).tolist(), rng.integers(0, 2 ** 31 - 1, 8191).tolist()]
    text = "\n".join(" ".join(map(str, [len(c)] + c)) for c in cases)
    out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.splitlines()
    for c, line in zip(cases, out):
        want = min(sum(c), top)
        assert line.split() == [str(want)] * 2
