"""Per-system kinetic energies at the sizes where their sums are cut into chunks of 512 bodies and free
atoms; alone and mixed in one batch. (The potential energies' chunks of 2048 units are covered by
test_gpu_forces.py, whose mixed box has 3600.)

Tolerance: the kinetic energies are FP64 sums over the body state; the comparison forms them from the
atoms' velocities, which mixed precision rounds in FP32 relative to the body (6e-8 of an atom's
velocity, so at most 2.4e-7 of the energy; held to 1e-6)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [[1], [511], [512], [513], [2048], [2049], [3, 1100, 512, 2100, 1]])
def test_kinetic_energies_of_systems_of_every_size(counts):
    from openmm_rigidbody_plugin_gb300 import batch, build
    from openmm_rigidbody_plugin_gb300 import workloads as W
    build.build_library()
    rng = np.random.default_rng(sum(counts))
    mass, body, x, v, box, q, s, e = [], [], [], [], [], [], [], []
    for n in counts:  # n waters and free atoms, one in five a free atom
        free = n // 5
        edge = max(2.2, (n * 0.035) ** (1 / 3))
        sites = W._lattice(n, edge)[rng.permutation(n)]
        rot = W.random_rotations(rng, n - free)
        wat = sites[:n - free, None, :] + np.einsum("aj,kij->kai", W.water_template(), rot)
        x.append(np.concatenate([wat.reshape(-1, 3), sites[n - free:]]))
        mass.append(np.concatenate([np.tile(W.WATER_MASSES, n - free), np.full(free, W.ARGON_MASS)]))
        body.append(np.concatenate([np.repeat(np.arange(1, n - free + 1), 3), np.zeros(free)]).astype(np.int32))
        q.append(np.concatenate([np.tile(W.WATER_CHARGES, n - free), np.zeros(free)]))
        s.append(np.concatenate([np.tile([W.WATER_SIGMA, 1.0, 1.0], n - free), np.full(free, W.ARGON_SIGMA)]))
        e.append(np.concatenate([np.tile([W.WATER_EPSILON, 0.0, 0.0], n - free), np.full(free, W.ARGON_EPSILON)]))
        v.append(rng.standard_normal((len(mass[-1]), 3)))
        box.append(edge)
    off = np.concatenate([[0], np.cumsum([len(m) for m in mass])])
    cut = [min(0.9, 0.49 * L) for L in box]
    mass, body, x, v, q, s, e = map(np.concatenate, (mass, body, x, v, q, s, e))
    b = batch.BatchedSystems(mass, body, off, box, cut, q, s, e)
    b.set_state(x, v)
    b.step(1, 0.0005)
    got = b.energies()
    _, v1 = b.get_state()
    for k in range(len(counts)):
        a = slice(off[k], off[k + 1])
        ke = 0.5 * float((mass[a, None] * v1[a] ** 2).sum())
        assert abs(got[k, 1] + got[k, 2] - ke) <= 1e-6 * ke, (counts[k], got[k], ke)
