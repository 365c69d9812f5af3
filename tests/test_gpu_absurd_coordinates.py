"""Coordinates too large to have a place in the box (FP32 leaves nothing of them modulo its edge) are accepted as
before: the call returns finite forces, and a system beside it is untouched bit for bit. The index arithmetic is checked on the CPU (test_list_cells.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edge,per_edge", [(4.375, 11), (8.375, 15), (4.0, 3), (2.0, 5)])
def test_absurd_coordinates_stay_with_their_system(edge, per_edge):
    from openmm_rigidbody_plugin_gb300 import batch, build
    build.build_library()
    rng = np.random.default_rng(per_edge)
    g = (np.arange(per_edge) + 0.5) * edge / per_edge
    one = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)
    one += 0.02 * rng.standard_normal(one.shape)
    n = len(one)

    def run(first):
        x = np.concatenate([first, one])
        b = batch.BatchedSystems(np.full(2 * n, 40.0), np.zeros(2 * n, dtype=np.int32), [0, n, 2 * n], [edge] * 2, [0.9] * 2,
                                 0.3 * (-1.0) ** np.arange(2 * n), np.full(2 * n, 0.2), np.full(2 * n, 0.5))
        b.set_state(x, np.zeros_like(x))
        f, u = b.forces()
        return f, u

    f, u = run(one)
    for big in (1e16, 5e16, -5e16, 1e18, 1e30):
        odd = one.copy()
        odd[n // 2, 0] = odd[3, 1] = odd[n - 1, 2] = big
        fo, uo = run(odd)
        assert np.array_equal(fo[n:], f[n:]) and uo[1] == u[1], big
        assert np.all(np.isfinite(fo))
