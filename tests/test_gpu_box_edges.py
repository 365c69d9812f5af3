"""Forces of atoms at the very edge of the periodic box, where FP32 wrapping may round a coordinate just
below zero to the box edge, or leave one just outside [0, L): every such atom keeps all of its neighbours,
and they keep it. Boxes whose list cells are half the reach (five an edge and more), the whole reach (three
and four an edge) and a single cell; one launch for small boxes and kernels over all units for large ones.

Tolerances, as in test_gpu_force_units.py: FP32 pair terms and sums from FP32 positions hold all atoms but
one in a thousand to 2e-5 of the largest force, and a pair within rounding of the cutoff, which may count on
one side only, moves an atom by at most 2e-3 of it; energies are held to 1e-5 kJ/mol per atom plus 1e-6.
Coordinates are given in FP32 and box edges are binary fractions, so that both sides wrap the same numbers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _argon(rng, edge, per_edge, places):
    """Argon with charges near a lattice; on each axis some atoms sit at the given coordinates."""
    g = (np.arange(per_edge) + 0.5) * edge / per_edge
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)
    x += 0.02 * rng.standard_normal(x.shape)
    n = len(x)
    for axis in range(3):  # the atoms of the first layer, spread over the face
        layer = np.nonzero(np.abs(x[:, axis] - g[0]) < 0.3 * edge / per_edge)[0]
        x[layer, axis] = np.resize(places, len(layer))
    corner = np.argmin(np.sum(x * x, axis=1))
    x[corner] = places[0]
    return x.astype(np.float32).astype(np.float64), 0.3 * (-1.0) ** np.arange(n)


@pytest.mark.parametrize("edge,per_edge,cutoff", [
    (2.75, 8, 0.9),      # 5 cells of half the reach
    (4.375, 11, 0.9),    # 8 of them
    (8.375, 15, 0.9),    # 16 of them
    (12.75, 20, 1.0),
    (4.0, 3, 0.9),       # sparse: three cells of the whole reach
    (5.25, 4, 0.9),      # sparse: five of them
    (2.0, 5, 0.9)])      # one cell
def test_atoms_at_the_box_edge_keep_their_neighbours(oracle_mod, edge, per_edge, cutoff):
    from openmm_rigidbody_plugin_gb300 import batch, build
    build.build_library()
    rng = np.random.default_rng(per_edge)
    below = np.nextafter(np.float32(edge), np.float32(0.0))
    places = [-1e-17, -1e-9, float(below), -1e-8, 0.0, edge, -1e-7, 10 * edge - 1e-6, 1e-9, -3 * edge, 1e-3]
    x, q = _argon(rng, edge, per_edge, places)
    n = len(x)
    s, e = np.full(n, 0.2), np.full(n, 0.5)
    body = np.zeros(n, dtype=np.int32)
    b = batch.BatchedSystems(np.full(n, 40.0), body, [0, n], [edge], [cutoff], q, s, e)
    b.set_state(x, np.zeros_like(x))
    pos, _ = b.get_state()
    f, u = b.forces()
    fo, uo = oracle_mod.lj_rf([0, n], [edge], [cutoff], pos, q, s, e, body)
    err = np.linalg.norm(f - fo, axis=1) / np.max(np.abs(fo))
    assert np.quantile(err, 1.0 - max(0.001, 1.5 / n)) < 2e-5 and np.max(err) < 2e-3, np.max(err)
    assert abs(u[0] - uo[0]) <= 1e-6 * abs(uo[0]) + 1e-5 * n, (u, uo)
