"""A body's step and a system's forces are the same bit for bit whatever else the handle holds: a body
beside one of more than 32 atoms (which selects another form of the step kernel) or, under NO-SQUISH, with
refined energies on; a system of few atom types beside others that together have too many for one
pair table."""
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


def _box(rng, edge, per_edge, types, sizes):
    """Bodies near a lattice, atom n of type n % types, types with charges of their own."""
    g = (np.arange(per_edge) + 0.5) * edge / per_edge
    at = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)
    size = np.resize(sizes, len(at))
    owner = np.repeat(np.arange(len(at)), size)
    n = len(owner)
    a = np.arange(n) - (np.cumsum(size) - size)[owner]
    x = at[owner] + 0.1 * np.stack([a % 2, a // 2 % 2, a // 4], axis=1) + 0.01 * rng.standard_normal((n, 3))
    t = np.arange(n) % types
    return (x, (owner + 1).astype(np.int32), 0.4 * np.cos(0.3 + 0.9 * np.pi * t / types), 0.2 + 0.001 * (t % 17),
            np.where(t % 3, 0.0, 0.2 + 0.003 * t))


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("types,sizes,edge,per_edge", [
    (3, [3], 3.0, 8),            # waters
    (12, [3, 4, 1, 6], 3.4, 8),  # units of one to four atoms
    (5, [3], 1.9, 5),            # one cell, the minimum image per pair
    (32, [2], 3.0, 8)])
def test_system_of_few_types_beside_one_of_many(types, sizes, edge, per_edge, precision):
    from openmm_rigidbody_plugin_gb300 import batch, build
    build.build_library()
    rng = np.random.default_rng(types)
    few, many = _box(rng, edge, per_edge, types, sizes), _box(rng, 3.2, 6, 77, [3, 5, 2])
    other = _box(rng, 4.2, 9, 31, [3])  # few types of its own, together more than 32

    def run(systems, edges):
        x, _, q, s, e = (np.concatenate(c) for c in zip(*systems))
        body = np.concatenate([w[1] + 10000 * i for i, w in enumerate(systems)]).astype(np.int32)
        off = np.concatenate([[0], np.cumsum([len(w[0]) for w in systems])])
        b = batch.BatchedSystems(np.full(len(x), 12.0), body, off, edges, [0.8] * len(systems), q, s, e, precision=precision)
        b.set_state(x, np.zeros_like(x))
        f, u = b.forces()
        b.relax(4)
        b.step(5, 0.001)
        xs, vs = b.get_state()
        n = off[1]
        return f[:n], u[0], xs[:n], vs[:n], b.energies()[0]

    alone = run([few], [edge])
    for beside in ([few, many], [few, other], [few, many, other]):
        edges = [edge] + [3.2 if w is many else 4.2 for w in beside[1:]]
        for a, b in zip(alone, run(beside, edges)):
            assert np.array_equal(a, b), np.abs(np.asarray(a) - np.asarray(b)).max()


@pytest.mark.parametrize("precision", ["mixed", "double"])
def test_waters_beside_units_of_other_sizes_and_in_batches_of_other_sizes(precision):
    """What a batch chooses for all of its systems (records per place, registers of the force pass, the set-up
    in one launch or in several) changes no system's bits."""
    from openmm_rigidbody_plugin_gb300 import batch, build
    build.build_library()
    rng = np.random.default_rng(8)
    waters = _box(rng, 3.0, 8, 3, [3])
    fours, singles, crowd = _box(rng, 3.0, 6, 5, [4]), _box(rng, 3.0, 7, 2, [1]), _box(rng, 6.2, 14, 3, [3])
    many = _box(rng, 3.2, 6, 77, [3, 5, 2])

    def run(systems, edges):
        x, _, q, s, e = (np.concatenate(c) for c in zip(*systems))
        body = np.concatenate([w[1] + 10000 * i for i, w in enumerate(systems)]).astype(np.int32)
        off = np.concatenate([[0], np.cumsum([len(w[0]) for w in systems])])
        b = batch.BatchedSystems(np.full(len(x), 12.0), body, off, edges, [0.8] * len(systems), q, s, e, precision=precision)
        b.set_state(x, np.zeros_like(x))
        f, u = b.forces()
        b.relax(4)
        b.step(5, 0.001)
        xs, vs = b.get_state()
        n = off[1]
        return f[:n], u[0], xs[:n], vs[:n], b.energies()[0]

    alone = run([waters], [3.0])
    for beside in ([(fours, 3.0)], [(singles, 3.0)], [(crowd, 6.2)], [(fours, 3.0), (crowd, 6.2)], [(many, 3.2), (crowd, 6.2)],
                   [(many, 3.2), (fours, 3.0)]):
        got = run([waters] + [w for w, _ in beside], [3.0] + [edge for _, edge in beside])
        for a, b in zip(alone, got):
            assert np.array_equal(a, b), np.abs(np.asarray(a) - np.asarray(b)).max()
