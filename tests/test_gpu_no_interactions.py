"""A batch without any interacting atom (no charges, no Lennard-Jones): zero forces and energies, ballistic
motion."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_batch_without_interactions():
    from openmm_rigidbody_plugin_gb300 import batch, build
    build.build_library()
    n = 40
    rng = np.random.default_rng(1)
    x, v = rng.uniform(0.0, 3.0, (2 * n, 3)), rng.standard_normal((2 * n, 3))
    zero = np.zeros(2 * n)
    free, half = np.zeros(2 * n, dtype=np.int32), [0, n, 2 * n]
    make = lambda q: batch.BatchedSystems(np.full(2 * n, 12.0), free, half, [3.0, 3.0], [0.9, 0.9], q, zero + 0.3, zero)  # noqa: E731
    used = [make(zero + q + 1.0) for q in range(24)]  # they leave their energies in the memory that they give back
    for b in used:
        b.set_state(x, v)
        assert np.all(b.forces()[1])
    kept, used, b = used[::4], None, None
    batches = [make(zero) for _ in range(12)]
    for b in batches:
        check(b, n, x, v)
    del kept


def check(b, n, x, v):
    b.set_state(x, v)
    f, u = b.forces()
    assert not np.any(f) and not np.any(u)
    kinetic = [6.0 * np.sum(v[k:k + n] ** 2) for k in (0, n)]
    b.step(4, 0.001)
    e = b.energies()
    assert not np.any(e[:, 0]) and not np.any(e[:, 2])
    assert np.allclose(e[:, 1], kinetic, rtol=1e-12, atol=0.0)
    assert np.abs(b.get_state()[0] - (x + 0.004 * v)).max() < 1e-12
