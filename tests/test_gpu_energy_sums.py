"""The pair energies of one unit are summed with compensation, each on its own: large ones that cancel
leave a small one whole. All coordinates are binary fractions and all pairs of the four atoms around
the fifth are at one distance, so equal and opposite charges give exactly opposite pair energies, and
what is left of a plain FP32 sum would be off by about a tenth of the small one.

Tolerance: the small pair energy is one FP32 product of factors rounded to FP32 (charges with their
constant, the reaction-field term whose parts are of its size): a few parts in 2^24 each, 2e-6 in all."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K = 138.935456


@pytest.mark.parametrize("types", [0, 40])  # with the pair table, and with more types than it holds
@pytest.mark.parametrize("arms", [3, 4])
def test_large_pair_energies_that_cancel(arms, types):
    from openmm_rigidbody_plugin_gb300 import batch, build
    build.build_library()
    edge, rc, r, eps = 16.0, 7.0, 3.0, 78.3
    centre = np.array([8.0, 8.0, 8.0])
    dirs = np.array([[1.0, 0, 0], [0, 1, 0], [0, 0, 1], [-1, 0, 0]])[:arms] * r
    big, small = 2.0 ** 11, 3.0 * 2.0 ** -12
    ring = np.array([big, small, -big, 0.0])[:arms]
    # body 1: the atoms around the centre; body 2: the charge at the centre and atoms out of reach of body 1
    far = np.array([[8.0, 8.0, 8.0], [0.0, 8.0, 8.0], [0.0, 0.0, 8.0], [0.0, 0.0, 0.0]])[:arms]
    x = np.concatenate([centre + dirs, far])
    q = np.concatenate([ring, [1.0], np.zeros(arms - 1)])
    tiny = 1e-30  # an interaction, too small to count
    e = np.concatenate([[0.0, 0.0, 0.0, tiny][:arms], [0.0] + [tiny] * (arms - 1)])
    s = np.full(len(x), 0.25)
    body = np.repeat([1, 2], arms).astype(np.int32)
    off, edges, cutoffs = [0, len(x)], [edge], [rc]
    if types:  # atoms of many types in the same box, without charges
        n = types
        lone = np.stack([np.full(n, 15.5), 2.0 + 0.01 * np.arange(n), np.full(n, 14.0)], axis=1)
        x, body = np.concatenate([x, lone]), np.concatenate([body, np.full(n, 3)]).astype(np.int32)
        q, s = np.concatenate([q, np.zeros(n)]), np.concatenate([s, 0.1 + 0.001 * np.arange(n)])
        e = np.concatenate([e, np.full(n, tiny)])
        off = [0, len(x)]
    b = batch.BatchedSystems(np.full(len(x), 12.0), body, off, edges, cutoffs, q, s, e, eps_solvent=eps,
                             precision="double")
    b.set_state(x, np.zeros_like(x))
    pos, _ = b.get_state()
    assert np.array_equal(pos[:arms + 1].astype(np.float32), x[:arms + 1]), "the positions are not exact"
    _, u = b.forces()
    krf = (eps - 1.0) / ((2.0 * eps + 1.0) * rc ** 3)
    one = K * small * (1.0 / r + krf * r * r - (1.0 / rc + krf * rc * rc))
    assert abs(u[0] - one) <= 2e-6 * abs(one), (u[0], one)
