"""The double-precision free rotation of an asymmetric top (csrc/rbx_math.cuh), compiled for the host and compared
with a fourth-order integration of the Euler equations in long double.

Error bounds. The body angular momentum is handed on as pi = 2 B(q) L and read back as Bt(q, pi)/2: two
rotations of four products each, and L(0) + dL before them, roundings of 2^-53 (|L| = 1) that add up to
1.6e-16 rms over the three components' largest error. Whatever else is rounded into it shows: two square
roots (each rounded to half an ulp or worse, and their product) make it 2.0e-16. The bound lies between,
1.85e-16, and the largest error at 1e-15. The quaternion is renormalised: 1.1e-16 rms, 4e-16 at most."""
import math
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

ROTATION = r"""
#include <algorithm>
#include <cstdio>
#include <random>
#include "rbx_math.cuh"
using namespace rbx;
typedef long double LD;

// one step of a seeded asymmetric top; the largest errors of q and of L (relative to |L|)
static void one(std::mt19937_64& g, double dt, int kind, double& eq, double& eL) {
    std::normal_distribution<double> N;
    std::uniform_real_distribution<double> U;
    double I[3];
    do {
        for (double& x : I) x = std::exp(3 * U(g) - 3);
        std::sort(I, I + 3, [](double a, double b) { return a > b; });
    } while (I[0] > I[1] + I[2] || I[0] - I[1] < 1e-3 * I[0] || I[1] - I[2] < 1e-3 * I[0]);
    double L[3];
    for (int k = 0; k < 3; k++) L[k] = N(g) * std::sqrt(I[k]) * 1.6;
    if (kind == 1) { L[1] *= 1e-5; L[2] *= 1e-5; }  // close to a principal axis
    if (kind == 2) { L[0] *= 1e-5; L[1] *= 1e-5; }
    if (kind == 3) { L[0] *= 1e-4; L[2] *= 1e-4; }
    const V3<double> i3 = v3<double>(I[0], I[1], I[2]), inv = v3<double>(1 / I[0], 1 / I[1], 1 / I[2]);
    Q4<double> q = q4<double>(N(g), N(g), N(g), N(g));
    q = q * (1 / std::sqrt(dot(q, q)));
    Q4<double> pi = qB(q, v3<double>(L[0], L[1], L[2])) * 2.0;
    LD y[7] = {q.w, q.x, q.y, q.z};
    const LD P[4] = {pi.w, pi.x, pi.y, pi.z};
    y[4] = 0.5L * (-y[1] * P[0] + y[0] * P[1] + y[3] * P[2] - y[2] * P[3]);
    y[5] = 0.5L * (-y[2] * P[0] - y[3] * P[1] + y[0] * P[2] + y[1] * P[3]);
    y[6] = 0.5L * (-y[3] * P[0] + y[2] * P[1] - y[1] * P[2] + y[0] * P[3]);
    auto rate = [&](const LD* a, LD* d) {
        LD w[3];
        for (int k = 0; k < 3; k++) w[k] = a[4 + k] / (LD)I[k];
        d[0] = -0.5L * (a[1] * w[0] + a[2] * w[1] + a[3] * w[2]);
        d[1] = 0.5L * (a[0] * w[0] + a[2] * w[2] - a[3] * w[1]);
        d[2] = 0.5L * (a[0] * w[1] + a[3] * w[0] - a[1] * w[2]);
        d[3] = 0.5L * (a[0] * w[2] + a[1] * w[1] - a[2] * w[0]);
        d[4] = a[5] * w[2] - a[6] * w[1];
        d[5] = a[6] * w[0] - a[4] * w[2];
        d[6] = a[4] * w[1] - a[5] * w[0];
    };
    const int S = 400;
    const LD h = (LD)dt / S;
    for (int s = 0; s < S; s++) {
        LD k1[7], k2[7], k3[7], k4[7], z[7];
        rate(y, k1);
        for (int i = 0; i < 7; i++) z[i] = y[i] + 0.5L * h * k1[i];
        rate(z, k2);
        for (int i = 0; i < 7; i++) z[i] = y[i] + 0.5L * h * k2[i];
        rate(z, k3);
        for (int i = 0; i < 7; i++) z[i] = y[i] + h * k3[i];
        rate(z, k4);
        for (int i = 0; i < 7; i++) y[i] += h / 6 * (k1[i] + 2 * k2[i] + 2 * k3[i] + k4[i]);
    }
    const LD n = sqrtl(y[0] * y[0] + y[1] * y[1] + y[2] * y[2] + y[3] * y[3]);
    exact_rotation_increment(i3, inv, q, pi, dt);
    const V3<double> l = qBt(q, pi) * 0.5;
    eq = (double)std::max({fabsl(q.w - y[0] / n), fabsl(q.x - y[1] / n), fabsl(q.y - y[2] / n), fabsl(q.z - y[3] / n)});
    eL = (double)std::max({fabsl(l.x - y[4]), fabsl(l.y - y[5]), fabsl(l.z - y[6])}) / std::sqrt(dot(l, l));
}

int main() {
    std::mt19937_64 g(7);
    for (double dt : {0.002, 0.01})
        for (int kind = 0; kind < 4; kind++) {
            double mq = 0, mL = 0, sq = 0, sL = 0;
            const int n = 1000;
            for (int t = 0; t < n; t++) {
                double eq, eL;
                one(g, dt, kind, eq, eL);
                mq = std::max(mq, eq); mL = std::max(mL, eL);
                sq += eq * eq; sL += eL * eL;
            }
            printf("%g %d %.4g %.4g %.4g %.4g\n", dt, kind, mq, std::sqrt(sq / n), mL, std::sqrt(sL / n));
        }
    return 0;
}
"""


def run(tmp_path, code):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    src, exe = tmp_path / "driver.cpp", tmp_path / "driver"
    src.write_text(code)
    csrc = os.path.join(ROOT, "openmm_rigidbody_plugin_gb300", "csrc")
    subprocess.run([gxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-I", csrc, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    return [[float(v) for v in line.split()] for line in out.splitlines()]


def test_error_of_one_step(tmp_path):
    rows = run(tmp_path, ROTATION)
    assert len(rows) == 8
    for dt, kind, mq, rq, mL, rL in rows:
        assert mq < 4e-16 and rq < 1.1e-16, (dt, kind, mq, rq)
        assert mL < 1e-15, (dt, kind, mL)
    mean = (sum(r[5] ** 2 for r in rows) / len(rows)) ** 0.5
    assert mean < 1.85e-16, mean


JACOBI = r"""
#include <algorithm>
#include <cstdio>
#include "rbx_math.cuh"
using namespace rbx;
typedef long double LD;

// sn, cn, dn by the arithmetic-geometric mean (Abramowitz & Stegun 16.4) in long double
static void agm(LD u, LD m1, LD* f) {  // m1 = 1 - m
    LD a[40], c[40], b = sqrtl(m1);
    a[0] = 1; c[0] = sqrtl(1 - m1);
    int n = 0;
    while (fabsl(c[n]) > 1e-19L && n < 30) {
        a[n + 1] = 0.5L * (a[n] + b);
        c[n + 1] = 0.5L * (a[n] - b);
        b = sqrtl(a[n] * b);
        n++;
    }
    LD phi = ldexpl(a[n] * u, n);
    for (; n > 0; n--) phi = 0.5L * (phi + asinl(c[n] / a[n] * sinl(phi)));
    f[0] = sinl(phi); f[1] = cosl(phi);
    f[2] = sqrtl(m1 + (1 - m1) * f[1] * f[1]);
}

int main() {
    for (double m1 : {0.99, 0.5, 0.1, 0.01, 1e-4, 1e-6, 1e-10})
        for (double h : {1e-3, 0.02, 0.031, 0.06, 0.12, 0.25, 0.4999, 0.5001, 0.9, 1.7, 3.0, 7.0, 20.0, 100.0, 600.0, 1e4, 1e6, 1e12}) {
            const double m = 1.0 - m1;
            LD f[3];
            agm(h, 1.0L - (LD)m, f);
            double s, c, d, n, sn, cm1, dm1;
            jacobi_homogeneous(h, m, s, c, d, n);
            jacobi_small_t(h, m, sn, cm1, dm1);
            const double e = (double)std::max({fabsl(s / (LD)n - f[0]), fabsl(c / (LD)n - f[1]), fabsl(d / (LD)n - f[2])});
            const double r = (double)std::max({fabsl(sn - f[0]), fabsl(1 + (LD)cm1 - f[1]), fabsl(1 + (LD)dm1 - f[2])});
            printf("%g %g %g %g\n", m1, h, e, r);
        }
    return 0;
}
"""


def test_jacobi_functions_in_homogeneous_coordinates(tmp_path):
    """sn, cn, dn as the quadrature takes them, of any argument, also next to the separatrix (1 - m from 0.99 to
    1e-10), against the arithmetic-geometric mean in long double. Each of the k duplications from below 1/32
    doubles the roundings (2^-53) before it, 2^k x 2^-53; beyond an argument h of 1/2 the quadrature itself is
    off by 4e-13 h^10, and the functions need be no better. They are finite wherever the form that divides at
    each duplication is."""
    rows = run(tmp_path, JACOBI)
    assert len(rows) == 7 * 18
    for m1, h, error, divided in rows:
        k = max(0, math.ceil(math.log2(h * 32)))
        assert error == error or divided != divided, (m1, h)
        if h <= 3.0:
            assert error <= max(2.0 ** (k - 53), 4e-13 * h ** 10), (m1, h, error)
