"""Forces and energies of waters (units of three atoms of which one has Lennard-Jones, or none) on both
sides of the number of atom types that a pair table holds: 32 types, and 33 or more, where each pair's
coefficients come from the two atoms. Two systems in a batch, bodies of four and five atoms among them,
against the FP64 all-pairs oracle.

Tolerances, as in test_gpu_force_units.py: FP32 pair terms and sums from FP32 positions hold 99.9 % of the
atoms to 2e-5 of the largest force, and a pair within rounding of the cutoff, which may count on one
side only, moves an atom by at most 2e-3 of it; energies are held to 1e-5 kJ/mol per atom plus 1e-6.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(rng, sizes, edge, types):
    """Bodies of the given sizes on a lattice; atom n has type n % types, whose charge is its own. Every
    third type has Lennard-Jones, every seventh body none."""
    k = int(np.ceil(len(sizes) ** (1 / 3)))
    g = (np.arange(k) + 0.5) * edge / k
    sites = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)[:len(sizes)]
    n = int(np.sum(sizes))
    owner = np.repeat(np.arange(len(sizes)), sizes)
    t = np.arange(n) % types
    a = np.arange(n) - (np.cumsum(sizes) - sizes)[owner]
    x = sites[owner] + 0.1 * np.stack([a % 2, a // 2 % 2, a // 4], axis=1) + 0.004 * rng.standard_normal((n, 3))
    charge = 0.4 * np.cos(1.0 + 0.9 * np.pi * t / types)
    sigma = 0.22 + 0.002 * (t % 5)
    eps = np.where((t % 3 == 0) & (owner % 7 != 3), 0.3 + 0.01 * (t % 7), 0.0)
    return x, owner + 1, charge, sigma, eps


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("sizes", [[3] * 300, [3] * 150 + [4] * 60 + [5] * 30])
@pytest.mark.parametrize("types", [18, 33, 257])  # 18 with and without Lennard-Jones are at most 32
def test_waters_of_few_and_many_types(oracle_mod, types, sizes, precision):
    from openmm_rigidbody_plugin_gb300 import batch, build
    build.build_library()
    rng = np.random.default_rng(types + len(sizes))
    one = _system(rng, np.array(sizes), 4.0, types)
    two = _system(rng, np.array([3] * 64), 2.2, types)
    x, body, q, s, e = (np.concatenate(c) for c in zip(one, two))
    body[len(one[0]):] += body[:len(one[0])].max()
    offsets, edges, cutoffs = [0, len(one[0]), len(x)], [4.0, 2.2], [0.9, 0.8]
    body = body.astype(np.int32)
    b = batch.BatchedSystems(np.full(len(x), 12.0), body, offsets, edges, cutoffs, q, s, e, precision=precision)
    b.set_state(x, np.zeros_like(x))
    for step in range(2):
        pos, _ = b.get_state()
        f, u = b.forces()
        fo, uo = oracle_mod.lj_rf(offsets, edges, cutoffs, pos, q, s, e, body)
        for i, (k, m) in enumerate(zip(offsets, offsets[1:])):
            err = np.linalg.norm(f[k:m] - fo[k:m], axis=1) / np.max(np.abs(fo[k:m]))
            assert np.quantile(err, 1.0 - 1.5 / (m - k)) < 2e-5 and np.max(err) < 2e-3, (i, step, np.max(err))
            assert abs(u[i] - uo[i]) <= 1e-6 * abs(uo[i]) + 1e-5 * (m - k), (i, u[i], uo[i])
        b.relax(3)
