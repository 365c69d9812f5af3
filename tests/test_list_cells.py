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
