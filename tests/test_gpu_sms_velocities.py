"""The SMS force where velocities differ much more across a scene than between
neighbours: fast particles among slow ones, and two halves that slide along
each other at the velocity limit. Every particle's force stays within the
rounding of its own pair terms (64 roundings of their magnitudes' sum, the
bound of the parity tests without its relative part): a slow particle's
viscosity does not lose its small velocity differences to a fast neighbour's
velocity."""
import numpy as np
import pytest

from gpu_helpers import dense_scene, shuffled

pytestmark = pytest.mark.gpu

FORCE_SUM_TOL = 64 * 2.0 ** -24


def velocities(field, pos, rng):
    v = rng.normal(0.0, 1e-3, (len(pos), 3))
    if field == "fast among slow":
        fast = rng.random(len(pos)) < 0.02
        v[fast] = rng.normal(0.0, 20.0, (fast.sum(), 3))
    else:
        v += 36.0 * np.sign(pos[:, 1:2] - np.median(pos[:, 1]))
    return v


@pytest.mark.parametrize("artificial", [None, (0.02, 20.0)])
@pytest.mark.parametrize("field", ["fast among slow", "sliding halves"])
def test_small_velocity_differences_survive(gsph, oracle, cuda_device, field, artificial):
    _, p, pos = dense_scene(gsph, n_side=30)
    with gsph.HybridSystem(params=p, positions=shuffled(pos)) as h:
        if artificial:
            h.set_viscosity_model(gsph.VISCOSITY_ARTIFICIAL, *artificial)
        h.arrange()
        h.density()
        q = h.copy_out(gsph.FIELD_POSITION)
        ev = h.copy_out(gsph.FIELD_EVAL_VELOCITY)
        ev[:, :3] = velocities(field, q, np.random.default_rng(7))
        h.copy_in(gsph.FIELD_EVAL_VELOCITY, ev)
        h.force()
        acc = h.copy_out(gsph.FIELD_ACCELERATION)[:, :3].astype(np.float64)
        key, start = h.copy_out(gsph.FIELD_KEY), h.copy_out(gsph.FIELD_CELL_START)
        assert h.info().tra_particles == 0
    force, mag = oracle.force(q, ev, key, start, p, with_mag=True, artificial=artificial)
    dev = np.linalg.norm(acc - force, axis=1)
    assert np.all(dev <= FORCE_SUM_TOL * mag), (dev / mag).max()
