"""The order in which the flat half steps correct a cell's absorbing layers
(fdtd_order.hpp, compiled here with the host compiler), for every way of
registering up to six layers: each cell meets at most one layer per axis, and
those have to come in registration order."""

import itertools
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fdtd_gb300", "csrc")

HARNESS = r"""
#include <cstdio>
#include "fdtd_order.hpp"
int main() {
    int n;
    while (scanf("%d", &n) == 1) {
        int axis[6] = {0}, high[6] = {0};
        for (int s = 0; s < n; ++s)
            if (scanf("%d %d", &axis[s], &high[s]) != 2) return 1;
        fdtd::LayerRank rank;
        const int order = fdtd::layer_order(n, axis, high, rank);
        printf("%d %d", order != fdtd::kOrderBySide, order);
        for (int c = 0; c < 8; ++c) printf(" %d", fdtd::cell_order(rank, c & 1, c & 2, c & 4));
        printf("\n");
    }
}
"""


def registrations():
    sides = [(a, h) for a in range(3) for h in range(2)]
    for n in range(7):
        yield from itertools.permutations(sides, n)


def axes_of(order):
    return [order >> 4 * r & 15 for r in range(3)]


@pytest.fixture(scope="module")
def orders(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("order")
    src, exe = d / "order.cpp", d / "order"
    src.write_text(HARNESS)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    regs = list(registrations())
    text = "".join(f"{len(r)} " + " ".join(f"{a} {h}" for a, h in r) + "\n" for r in regs)
    out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout
    return list(zip(regs, [[int(v) for v in line.split()] for line in out.splitlines()]))


def test_one_order_is_a_registration_order(orders):
    assert len(orders) == 1957
    for reg, (one, order, *_) in orders:
        if not one:
            continue
        got = axes_of(order)
        assert sorted(got) == [0, 1, 2]
        for s, t in itertools.combinations(reg, 2):
            assert s[0] == t[0] or got.index(s[0]) < got.index(t[0]), (reg, order)


def test_order_of_a_cell_by_its_sides(orders):
    """Layers of two axes that interleave: a cell's own layers in registration
    order, whichever side of each axis it is on."""
    sides = list(itertools.product(range(2), repeat=3))
    assert any(not one for _, (one, *_) in orders)
    for reg, (_, _, *cells) in orders:
        for z, y, x in sides:
            got = axes_of(cells[x + 2 * y + 4 * z])
            assert sorted(got) == [0, 1, 2]
            mine = [a for a, h in reg if h == (x, y, z)[a]]
            assert [a for a in got if a in mine] == mine, (reg, got)


def test_plain_order_wherever_the_layers_allow_it(orders):
    """x, y, z is unrolled in the kernels; axes without a layer do not count."""
    for reg, (one, order, *_) in orders:
        axes = [a for a, _ in reg]
        if axes == sorted(axes):
            assert one and axes_of(order) == [0, 1, 2], (reg, order)
