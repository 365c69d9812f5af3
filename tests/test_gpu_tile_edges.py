"""The step at body counts around warp and tile edges, all rotation classes in random order, against the
robust FP64 oracle: how bodies are packed into tiles (as few whole warps as fill a wave) and, in
double precision, taken by rotation class changes with the count, and no body's result may.

Tolerances as in test_gpu_parity_degenerate.py (there after 100 steps, here after 20): positions,
velocities and kinetic energies, double 1e-9, 1e-8, 1e-9; mixed 1e-6, 1.5e-6, 1e-6. A count of thousands
compares with the same bodies in a system of their own, bit for bit (bodies do not interact here)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"double": (1e-9, 1e-8, 1e-9), "mixed": (1e-6, 1.5e-6, 1e-6)}


def _run(masses, bidx, x, v, f, mode, prec, steps):
    from openmm_rigidbody_plugin_gb300 import build, kernel
    build.build_library()
    k = kernel.IntegratorKernel(masses, bidx, rotation_mode=mode, precision=prec)
    buf = kernel.DeviceBuffers(len(masses), precision=prec)
    buf.set_positions(x)
    buf.set_velocities(v, masses)
    buf.set_forces(f)
    k.upload_state_device(buf)
    k.part1(buf, 0.002)
    for _ in range(steps - 1):
        k.fused(buf, 0.002)
    k.part2(buf, 0.002)
    return buf.get_positions(), buf.get_velocities(), k.kinetic_energies(buf)


@pytest.mark.parametrize("prec", ["mixed", "double"])
@pytest.mark.parametrize("mode", [0, 4])
@pytest.mark.parametrize("n,free", [(1, 0), (31, 1), (33, 0), (97, 257), (130, 3), (0, 40)])
def test_small_counts_match_the_oracle(oracle_mod, n, free, mode, prec):
    from openmm_rigidbody_plugin_gb300 import workloads as W
    s = W.mixed_system(n_bodies=n, n_free=free, fractions=(0.5, 0.3, 0.2) if n > 1 else (1.0, 0.0, 0.0), seed=n + free)
    f = np.round(W.gaussian_forces(s.num_atoms, seed=5, sd=50.0) * 2.0 ** 32) / 2.0 ** 32
    x, v, ke = _run(s.masses, s.body_indices, s.positions, s.velocities, f, mode, prec, 20)
    o = oracle_mod.Oracle(s.masses, s.body_indices, mode=mode, robust=True)
    o.setup(s.positions, s.velocities, f)
    for _ in range(20):
        o.part1(0.002, f)
        o.part2(0.002, f)
    for a, b, tol in zip((x, v, ke), (o.R, o.V, np.array(o.kinetic())), TOL[prec]):
        assert np.abs(a - b).max() <= tol * np.abs(b).max(), (n, free, np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("prec", ["single", "mixed", "double"])
@pytest.mark.parametrize("mode", [0, 4])
def test_bodies_of_a_large_system_equal_themselves_in_a_small_one(mode, prec):
    from openmm_rigidbody_plugin_gb300 import workloads as W
    s = W.mixed_system(n_bodies=30011, n_free=777, seed=4)
    f = W.gaussian_forces(s.num_atoms, seed=5, sd=50.0)
    x, v, _ = _run(s.masses, s.body_indices, s.positions, s.velocities, f, mode, prec, 3)
    keep = (s.body_indices == 0) | (s.body_indices % 97 == 0)
    xs, vs, _ = _run(s.masses[keep], s.body_indices[keep], s.positions[keep], s.velocities[keep], f[keep], mode, prec, 3)
    assert np.array_equal(x[keep], xs) and np.array_equal(v[keep], vs)
