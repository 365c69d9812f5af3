"""Forces and energies of rigid bodies of many sizes against the FP64 all-pairs oracle, at the sizes where
the force pass changes form: bodies of 1 to 4 atoms (one unit of neighbour lists), 5, 8, 13 and 45
(several units), bodies with and without Lennard-Jones on their last atoms, atoms without any
interaction between them, few atom types (pair table) and more than 32, boxes of one list cell (with
and without the minimum image per pair), of cells of half the reach (five an edge and more) and, where
sparse, of the whole reach (three and more).

Tolerances, as in test_gpu_forces.py: FP32 pair terms and sums from FP32 positions hold 99.9 % of the
atoms to 2e-5 of the largest force, and a pair within rounding of the cutoff, which may count on one
side only, moves an atom by at most 2e-3 of it; energies are held to 1e-5 kJ/mol per atom plus 1e-6.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _box(rng, sizes, edge, types):
    """Compact rigid bodies of the given sizes on a lattice, in random order; every third atom past
    a body's first has charge only, and every seventh atom of the larger bodies nothing."""
    k = int(np.ceil(len(sizes) ** (1 / 3)))
    g = (np.arange(k) + 0.5) * edge / k
    sites = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)
    sites = sites[rng.permutation(len(sites))[:len(sizes)]]
    x, body, charge, sigma, eps = [], [], [], [], []
    n = 0
    for b, size in enumerate(rng.permutation(sizes)):
        m = int(np.ceil(size ** (1 / 3)))
        h = (np.arange(m) - 0.5 * (m - 1)) * 0.1
        cloud = np.stack(np.meshgrid(h, h, h, indexing="ij"), axis=-1).reshape(-1, 3)[:size]
        x.append(sites[b] + cloud + 0.004 * rng.standard_normal((size, 3)))
        for a in range(size):
            t = n % types
            bare = a > 0 and a % 3 == 0
            mute = size > 4 and a % 7 == 6
            body.append(b + 1 if size > 1 else 0)
            charge.append(0.0 if mute else 0.3 * np.cos(2.1 * t))
            sigma.append(0.2 + 0.002 * (t % 5))
            eps.append(0.0 if bare or mute else 0.2 + 0.01 * (t % 7))
            n += 1
    return (np.concatenate(x), np.array(body, dtype=np.int32), np.array(charge), np.array(sigma), np.array(eps))


@pytest.mark.parametrize("types", [5, 200])
@pytest.mark.parametrize("name,sizes,edge,cutoff", [
    ("singles", [1] * 200, 2.4, 0.8),
    ("pairs", [2] * 150, 2.4, 0.7),
    ("threes in a box at half the cutoff", [3] * 64, 1.9, 0.93),
    ("threes", [3] * 400, 4.4, 0.8),
    ("fours", [4] * 300, 4.6, 0.9),
    ("many", [1] * 90 + [2] * 60 + [3] * 120 + [4] * 40 + [5] * 30 + [8] * 20 + [13] * 6 + [45] * 2, 5.2, 0.85),
    ("sparse", [3] * 60, 7.0, 0.8),
    ("sparse, three cells an edge", [1] * 30 + [3] * 30 + [8] * 4, 4.0, 0.9),
    ("one body and one atom", [45, 1], 2.2, 0.9)])
def test_forces_of_bodies_of_every_size(oracle_mod, name, sizes, edge, cutoff, types):
    from openmm_rigidbody_plugin_gb300 import batch, build
    build.build_library()
    rng = np.random.default_rng(len(sizes) + types)
    x, body, q, s, e = _box(rng, np.array(sizes), edge, types)
    masses = np.full(len(x), 12.0)
    b = batch.BatchedSystems(masses, body, [0, len(x)], [edge], [cutoff], q, s, e)
    b.set_state(x, np.zeros_like(x))
    for step in range(2):
        pos, _ = b.get_state()
        f, u = b.forces()
        fo, uo = oracle_mod.lj_rf([0, len(x)], [edge], [cutoff], pos, q, s, e, body)
        err = np.linalg.norm(f - fo, axis=1) / (np.max(np.abs(fo)) or 1.0)  # bodies may lie out of reach
        assert np.quantile(err, 0.999 if len(x) > 1000 else 1.0 - 1.5 / len(x)) < 2e-5 and np.max(err) < 2e-3, (
            name, step, np.max(err))
        assert np.all(np.abs(u - uo) <= 1e-6 * np.abs(uo) + 1e-5 * len(x)), (name, u, uo)
        b.relax(3)  # other positions, lists built on the way
