"""How the points of a soft source are grouped (fdtd_groups.hpp, compiled here
with the host compiler): lines along an axis and full boxes stay whole, and no
group's bounding box holds more than eight cells per point, so a diagonal line
does not send every cell of the grid looking for a point."""

import itertools
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fdtd_gb300", "csrc")

HARNESS = r"""
#include <cstdio>
#include <vector>
#include "fdtd_groups.hpp"
int main() {
    int n;
    while (scanf("%d", &n) == 1) {
        std::vector<int> x(3 * n);
        for (int &v : x)
            if (scanf("%d", &v) != 1) return 1;
        for (int q = 0; q < n;) {
            q = fdtd::group_end(q, n, [&](int p, int a) { return x[3 * p + a]; });
            printf("%d ", q);
        }
        printf("\n");
    }
}
"""


def _sorted(points):
    return sorted(tuple(int(v) for v in p) for p in points)


def _cases():
    yield "line x", [(q, 3, 4) for q in range(50)], 1
    yield "line z", [(2, 3, q) for q in range(500)], 1
    yield "every third cell", [(2, 3 * q, 4) for q in range(60)], 1
    yield "box", list(itertools.product(range(3), range(4), range(5))), 1
    yield "plane", list(itertools.product(range(9), [3], range(7))), 1
    yield "one cell, often", [(1, 2, 3)] * 9, 1
    yield "two far points", [(0, 0, 0), (90, 80, 70)], 2
    yield "diagonal 2d", [(q, q, 0) for q in range(400)], None
    yield "diagonal 3d", [(q, q, q) for q in range(100)], None
    yield "slope", [(q, q // 40, 0) for q in range(500)], None
    rng = np.random.default_rng(5)
    for _ in range(60):
        hi = rng.integers(1, 40, size=3)
        yield "random", list(map(tuple, rng.integers(0, hi, size=(int(rng.integers(2, 80)), 3)))), None


def test_groups():
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host compiler")
    cases = [(name, _sorted(p), n) for name, p, n in _cases()]
    import tempfile

    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "groups.cpp"), os.path.join(d, "groups")
        open(src, "w").write(HARNESS)
        subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-I", CSRC, src, "-o", exe], check=True)
        text = "\n".join(f"{len(p)} " + " ".join(str(v) for q in p for v in q) for _, p, _ in cases) + "\n"
        out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout
    for (name, points, groups), line in zip(cases, out.splitlines(), strict=True):
        ends = [int(v) for v in line.split()]
        assert ends[-1] == len(points) and ends == sorted(set(ends)), name
        for a, b in zip([0] + ends, ends):
            p = np.array(points[a:b])
            assert np.prod(p.max(0) - p.min(0) + 1) <= 8 * len(p), (name, a, b)
        if groups is not None:
            assert len(ends) == groups, name
