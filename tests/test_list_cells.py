"""Wrapping of coordinates into the periodic box and their list cells (csrc/rbx_cells.h), compiled for the host
and checked on the CPU: a wrapped coordinate lies in [0, L), is the given one up to whole box edges, and lies
in the cell that it is counted in. The neighbour search shifts whole cells, so a unit whose coordinate and cell
disagreed would miss all of its neighbours."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

DRIVER = r"""
#include <cstdio>
#include "rbx_cells.h"
int main() {  // lines of: x L nc -> wrapped cell
    float x, L;
    int nc;
    while (scanf("%a %a %d", &x, &L, &nc) == 3) {
        const float invL = (float)(1.0 / (double)L), c = rbx::wrap_coordinate(x, L, invL);
        printf("%a %d\n", c, rbx::cell_of(c, invL, nc));
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def wrap(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    d = tmp_path_factory.mktemp("cells")
    src, exe = d / "cells.cpp", d / "cells"
    src.write_text(DRIVER)
    csrc = os.path.join(ROOT, "openmm_rigidbody_plugin_gb300", "csrc")
    subprocess.run([gxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-I", csrc, str(src), "-o", str(exe)], check=True)

    def call(x, L, nc):
        lines = "".join(f"{float(a).hex()} {float(b).hex()} {int(k)}\n" for a, b, k in zip(x, L, nc))
        out = subprocess.run([str(exe)], input=lines, check=True, capture_output=True, text=True).stdout.split()
        return np.array([float.fromhex(v) for v in out[::2]]), np.array([int(v) for v in out[1::2]])
    return call


RANGES = r"""
#include <cstdio>
#include "rbx_cells.h"
int main() {  // lines of: x h L nc w -> the ranges of the parts that the search takes
    float x, h, L;
    int nc, w;
    while (scanf("%f %f %f %d %d", &x, &h, &L, &nc, &w) == 5) {
        const float invL = 1.0f / L;
        const int c = rbx::cell_of(x, invL, nc);
        const rbx::CellRange r = rbx::cells_within(x, h, invL * (float)nc, c, w);
        const int parts = c < w || c >= nc - w ? 2 : 1;
        printf("%d %d", c, parts);
        for (int p = 0; p < 2; p++) {
            const rbx::CellRange in = p < parts ? rbx::range_part(r, p, c, w, nc) : rbx::CellRange{0, -1};
            printf(" %d %d", in.a, in.b);
        }
        printf("\n");
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def ranges(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    d = tmp_path_factory.mktemp("ranges")
    src, exe = d / "ranges.cpp", d / "ranges"
    src.write_text(RANGES)
    csrc = os.path.join(ROOT, "openmm_rigidbody_plugin_gb300", "csrc")
    # signed overflow and conversions out of range end the program
    subprocess.run([gxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-fsanitize=undefined,float-cast-overflow",
                    "-fno-sanitize-recover=all", "-I", csrc, str(src), "-o", str(exe)], check=True)

    def call(cases):
        lines = "".join(" ".join(str(v) for v in c) + "\n" for c in cases)
        out = subprocess.run([str(exe)], input=lines, check=True, capture_output=True, text=True).stdout
        return np.array([[int(v) for v in line.split()] for line in out.splitlines()])
    return call


def test_cells_in_reach_are_taken_once_each(ranges):
    rng = np.random.default_rng(3)
    cases = []
    for _ in range(3000):
        w = int(rng.integers(1, 3))
        nc = int(rng.integers(2 * w + 1, 14))
        edge = float(rng.uniform(0.3, 2.0))
        cases.append((float(np.float32(rng.uniform(0, nc * edge * (1 - 1e-6)))), rng.uniform(0.0, w * edge), nc * edge, nc, w))
    out = ranges(cases)
    for (x, h, L, nc, w), (c, _, a0, b0, a1, b1) in zip(cases, out):
        taken = list(range(a0, b0 + 1)) + list(range(a1, b1 + 1))
        assert len(taken) == len(set(taken)) and all(0 <= k < nc for k in taken)
        edge, slack = L / nc, 1e-4
        met = {int(np.floor(t / edge)) % nc for t in np.arange(x - h + slack, x + h - slack, 0.01 * edge)}
        assert met <= set(taken), (x, h, L, nc, w, taken, met)


def test_coordinates_without_a_place_in_the_box_stay_in_the_cell_table(ranges):
    values = [s * v for s in (-1, 1) for v in (1e5, 1e8, 1.5e9, 2.2e9, 3e12, 1e30, 3e38, float("inf"))]
    reaches = [0.5, 1e6, 1e20, float("inf")]
    cases = [(x, h, L, nc, w) for x in values for h in reaches for L, nc, w in ((4.4, 7, 2), (3.0, 3, 1), (5.0, 5, 2))]
    for case, (c, _, a0, b0, a1, b1) in zip(cases, ranges(cases)):
        for a, b in ((a0, b0), (a1, b1)):
            assert a > b or (0 <= a and b < case[3]), (case, a, b)


def test_wrapped_coordinates_lie_in_their_cells(wrap):
    rng = np.random.default_rng(2)
    x, L, nc = [], [], []
    for edge in np.float32(np.concatenate([[2.9, 4.0, 4.4, 8.37, 12.8, 2.75, 1.0, 3.0], rng.uniform(1.5, 40.0, 60)])):
        e = float(edge)
        below, above = float(np.nextafter(edge, np.float32(0))), float(np.nextafter(edge, np.float32(99)))
        some = [0.0, -0.0, -1e-38, -1e-17, -1e-9, -1e-8, -1e-7, -1e-6, 1e-9, below, e, above, -below, -e, -above]
        some += [k * e + d for k in (-40, -10, -3, -1, 1, 2, 10, 40, 1000) for d in (-1e-5, -1e-6, -1e-7, 0.0, 1e-7, 1e-6)]
        some += list(rng.uniform(-3 * e, 3 * e, 60))
        x += some
        L += [e] * len(some)
        nc += list(rng.integers(3, max(4, int(e / 0.4)), len(some)))
    x, L, nc = np.float32(x).astype(float), np.array(L), np.array(nc)
    c, cell = wrap(x, L, nc)
    assert np.all((c >= 0.0) & (c < L)), (x[~((c >= 0) & (c < L))], c[~((c >= 0) & (c < L))])
    off = np.abs((x - c) / L - np.round((x - c) / L)) * L  # rounding of x and of L in FP32 only
    assert np.all(off <= 2.0 ** -23 * (np.abs(x) + L))
    assert np.all((cell >= 0) & (cell < nc))
    edge = L / nc
    assert np.all((cell * edge <= c + 1e-5) & (c - 1e-5 <= (cell + 1) * edge))
