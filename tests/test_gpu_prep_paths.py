"""The set-up of a force evaluation in one block per system (batches of systems of at most 1024 units) and
in kernels over all units (a batch with a larger one): the same places and lists, so a system's
trajectory, energies and list builds are the same bit for bit alone and beside a larger system, with
one list cell and with many."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,box", [(1, 2.5), (31, 2.2), (1024, None), (1024, 4.4), (700, 6.0), (1025, 4.4)])
def test_system_alone_equals_system_beside_a_large_one(n, box):
    from openmm_rigidbody_plugin_gb300 import batch, build
    from openmm_rigidbody_plugin_gb300 import workloads as W
    build.build_library()
    small = W.water_box(n, seed=n, box=box)
    large = W.water_box(1100, seed=2)
    alone = batch.BatchedSystems.from_systems([small])
    beside = batch.BatchedSystems.from_systems([large, small])
    for b in (alone, beside):
        b.relax(20)
        x, v = b.get_state()
        b.set_state(x, v)
        b.step(40, 0.002)
    a = alone.get_state()
    for k in range(2):
        assert np.array_equal(a[k], beside.get_system_state(1)[k])
    assert np.array_equal(alone.energies()[0], beside.energies()[1])
    assert alone.list_builds()[0] == beside.list_builds()[1]
    assert n == 1 or alone.list_builds()[0] > 4
