"""A body's step is the same bit for bit whatever else the handle holds: beside a body of more than 32 atoms
(which selects another form of the step kernel) and, under NO-SQUISH, with refined energies on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _steps(masses, bidx, x, v, f, mode, prec, refined=False, steps=12):
    from openmm_rigidbody_plugin_gb300 import build, kernel
    build.build_library()
    k = kernel.IntegratorKernel(masses, bidx, rotation_mode=mode, precision=prec)
    if refined:
        k.set_compute_refined_energies(True)
    buf = kernel.DeviceBuffers(len(masses), precision=prec)
    buf.set_positions(x)
    buf.set_velocities(v, masses)
    buf.set_forces(f)
    k.upload_state_device(buf)
    k.part1(buf, 0.002)
    for _ in range(steps - 1):
        k.fused(buf, 0.002)
    k.part2(buf, 0.002)
    n = len(masses)
    out = [buf.posq[:n].cpu().numpy(), buf.velm[:n].cpu().numpy()]
    return out + ([buf.corr[:n].cpu().numpy()] if buf.corr is not None else [])


@pytest.mark.parametrize("prec", ["single", "mixed", "double"])
@pytest.mark.parametrize("mode", [0, 1, 4])
def test_bodies_beside_a_large_one_and_with_refined_energies(mode, prec):
    from openmm_rigidbody_plugin_gb300 import workloads as W
    s = W.mixed_system(n_bodies=900, n_free=50, seed=3)
    f = W.gaussian_forces(s.num_atoms, seed=4, sd=50.0)
    rng = np.random.default_rng(9)
    m = 64  # one body of 64 atoms after the others
    masses = np.concatenate([s.masses, np.full(m, 12.0)])
    bidx = np.concatenate([s.body_indices, np.full(m, s.body_indices.max() + 1, dtype=np.int32)])
    x = np.concatenate([s.positions, 1.0 + 0.3 * rng.standard_normal((m, 3))])
    v = np.concatenate([s.velocities, rng.standard_normal((m, 3))])
    fl = np.concatenate([f, rng.standard_normal((m, 3))])
    n = s.num_atoms
    plain = _steps(s.masses, s.body_indices, s.positions, s.velocities, f, mode, prec)
    large = _steps(masses, bidx, x, v, fl, mode, prec)
    for a, b in zip(plain, large):
        assert np.array_equal(a, b[:n]), np.abs(a - b[:n]).max()
    if mode:  # (the exact rotation's refined form is compiled apart, and free atoms are then stepped in FP64)
        refined = _steps(s.masses, s.body_indices, s.positions, s.velocities, f, mode, prec, refined=True)
        bodies = s.body_indices > 0
        for a, b in zip(plain, refined):
            assert np.array_equal(a[bodies], b[bodies]), np.abs(a - b)[bodies].max()
