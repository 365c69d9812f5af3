"""Neighbour lists of systems that are not filled evenly, against the FP64 all-pairs oracle: clusters of
large rigid bodies (each many list entries) in a dilute box, a droplet of waters, and systems that have
grown far denser than the state their lists were sized for.

Tolerances, as in test_gpu_force_units.py: FP32 pair terms and sums from FP32 positions hold all atoms but
one in a thousand to 2e-5 of the largest force, and a pair within rounding of the cutoff, which may count on
one side only, moves an atom by at most 2e-3 of it; energies of the clusters, whose atoms are jittered, are
held to 1e-5 kJ/mol per atom plus 1e-6 (waters on a lattice repeat the same distances, and the rounding of
their pair energies then adds up instead of averaging out)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lattice(k, step):
    g = (np.arange(k) - 0.5 * (k - 1)) * step
    return np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)


class _System:
    """Rigid bodies of one kind about the centres `at` (which other states of them may share)."""

    def __init__(self, at, inner, charge, sigma, epsilon):
        self.at, self.inner, self.size = at, inner, inner.shape[1]
        n = len(at)
        self.x = (at[:, None, :] + inner).reshape(-1, 3)
        self.body = np.repeat(np.arange(n) + 1, self.size).astype(np.int32)
        self.q, self.s, self.e = (np.tile(c, n) for c in (charge, sigma, epsilon))

    def moved_to(self, at, time):
        """Velocities that take every body to the centre at[b] in the given time."""
        return np.repeat((at - self.at) / time, self.size, axis=0)


def _clusters(per_edge, gap, edge):
    """Rigid bodies of 4 x 4 x 4 atoms, per_edge^3 of them with the given gap between neighbours, about the
    centre of a box."""
    cube = _lattice(4, 0.14) * np.array([1.0, 1.02, 1.05])
    at = _lattice(per_edge, 3 * 0.14 * 1.05 + gap) + 0.5 * edge
    jitter = 0.003 * np.random.default_rng(per_edge).standard_normal((len(at), 64, 3))
    return _System(at, cube + jitter, 0.3 * np.cos(1.7 * np.arange(64)), np.full(64, 0.25), np.full(64, 0.3))


def _waters(per_edge, step, edge):
    from openmm_rigidbody_plugin_gb300 import workloads as W
    at = _lattice(per_edge, step) + 0.5 * edge
    rot = W.random_rotations(np.random.default_rng(per_edge), len(at))
    q, s, e = (np.array(c) for c in zip(*(W.NONBONDED[k] for k in W.SPECIES["water"])))
    return _System(at, np.einsum("bij,aj->bai", rot, W.TEMPLATES["water"]), q, s, e)


def _batch(systems, edge, cutoff, velocities=None, positions=None):
    from openmm_rigidbody_plugin_gb300 import batch, build
    build.build_library()
    off = np.concatenate([[0], np.cumsum([len(w.x) for w in systems])])
    body = np.concatenate([w.body + 10000 * i for i, w in enumerate(systems)]).astype(np.int32)
    x, q, s, e = (np.concatenate([getattr(w, c) for w in systems]) for c in "xqse")
    b = batch.BatchedSystems(np.full(len(x), 12.0), body, off, [edge] * len(systems), [cutoff] * len(systems), q, s, e)
    b.set_state(x if positions is None else positions, np.zeros_like(x) if velocities is None else velocities)
    return b


def _matches_oracle(oracle_mod, b, system, edge, cutoff):
    n = len(system.x)
    pos, _ = b.get_state()
    f, u = b.forces()
    fo, uo = oracle_mod.lj_rf([0, n], [edge], [cutoff], pos, system.q, system.s, system.e, system.body)
    err = np.linalg.norm(f - fo, axis=1) / (np.max(np.abs(fo)) or 1.0)  # wide states may have no pair in reach
    assert np.quantile(err, 1.0 - max(0.001, 1.5 / n)) < 2e-5 and np.max(err) < 2e-3, np.max(err)
    if system.size == 64:
        assert abs(u[0] - uo[0]) <= 1e-6 * abs(uo[0]) + 1e-5 * n, (u, uo)
    assert not np.any(b.status())


@pytest.mark.parametrize("name,per_edge,edge", [("eight bodies", 2, 10.0), ("eight bodies", 2, 4.0),
                                                ("27 bodies", 3, 12.0)])
def test_clusters_of_large_bodies_in_a_dilute_box(oracle_mod, name, per_edge, edge):
    system = _clusters(per_edge, 0.33, edge)
    _matches_oracle(oracle_mod, _batch([system], edge, 0.9), system, edge, 0.9)


@pytest.mark.parametrize("per_edge,edge", [(7, 9.0), (11, 20.0)])  # one block per system; all units
def test_droplet_of_waters(oracle_mod, per_edge, edge):
    system = _waters(per_edge, 0.32, edge)
    _matches_oracle(oracle_mod, _batch([system], edge, 0.9), system, edge, 0.9)


TIME = 0.01  # ps: short enough that forces move nothing by more than about 1e-4 nm


@pytest.mark.parametrize("kind", ["clusters", "waters", "waters in one cell"])
def test_state_far_denser_than_the_one_the_lists_were_sized_for(oracle_mod, kind):
    """The bodies fly together in one long step, and then back."""
    make, per_edge, far, near, edge, cutoff = {"clusters": (_clusters, 3, 3.0, 0.33, 12.0, 0.9),
                                               "waters": (_waters, 9, 1.7, 0.32, 16.0, 0.9),
                                               "waters in one cell": (_waters, 6, 0.69, 0.32, 4.375, 1.6)}[kind]
    wide, dense = make(per_edge, far, edge), make(per_edge, near, edge)
    b = _batch([wide], edge, cutoff, wide.moved_to(dense.at, TIME))
    _matches_oracle(oracle_mod, b, wide, edge, cutoff)
    b.step(1, TIME)
    assert np.abs(b.get_state()[0] - dense.x).max() < 0.01
    _matches_oracle(oracle_mod, b, dense, edge, cutoff)
    # and the forces that lists sized for this state give, up to the order of their sums
    f, u = b.forces()
    fc, uc = _batch([dense], edge, cutoff, positions=b.get_state()[0]).forces()
    assert np.abs(f - fc).max() <= 2e-5 * np.abs(fc).max() and abs(u[0] - uc[0]) <= 1e-6 * abs(uc[0]) + 1e-5 * len(f)
    b.step(1, -TIME)
    _matches_oracle(oracle_mod, b, wide, edge, cutoff)


def test_a_system_short_of_list_room_gives_the_same_alone_and_in_a_batch():
    """Its capacity is its own: not raised by a denser system beside it."""
    edge, cutoff = 9.0, 0.9
    wide, dense, crowd = _waters(7, 1.2, edge), _waters(7, 0.32, edge), _clusters(3, 0.33, edge)
    v = wide.moved_to(dense.at, TIME)
    alone = _batch([wide], edge, cutoff, v)
    beside = _batch([wide, crowd], edge, cutoff, np.concatenate([v, np.zeros_like(crowd.x)]))
    n = len(wide.x)
    for b in (alone, beside):
        b.step(1, TIME)
    for a, c in zip(alone.forces(), beside.forces()):
        assert np.array_equal(a, c[:len(a)])
    for a, c in zip(alone.get_state(), beside.get_state()):
        assert np.array_equal(a, c[:n])
