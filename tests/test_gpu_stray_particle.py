"""A particle far outside the grid is clamped into a boundary cell and reported;
the other particles of that cell keep their neighbours. In SMS cells the
candidates are tested against the bounding box of 16 particles, which such a
particle stretches until coordinate differences round by more than the kernel
radius: density and force of all others equal the FP64 oracle's for the scene
without it, as in TRA cells."""
import numpy as np
import pytest

from gpu_helpers import dense_scene, shuffled

pytestmark = pytest.mark.gpu

RHO_TOL = 1e-5
FORCE_TOL = 1e-4
FORCE_SUM_TOL = 64 * 2.0 ** -24


def run(gsph, p, pos):
    with gsph.HybridSystem(params=p, positions=pos) as h:
        h.arrange()
        h.density()
        h.force()
        perm = h.copy_out(gsph.FIELD_PERMUTATION)
        out = {f: h.copy_out(getattr(gsph, "FIELD_" + f)) for f in
               ("POSITION", "EVAL_VELOCITY", "ACCELERATION", "KEY", "CELL_START")}
        out["tasks"], out["perm"] = h.info().sms_tasks, perm
    return out


@pytest.mark.parametrize("away", [-5.0, -1e4, -6e5, -9e5, -1e9, -1e25])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_neighbours_of_a_stray_particle_keep_theirs(gsph, oracle, cuda_device, axis, away):
    _, p, block = dense_scene(gsph, n_side=14)
    block[:, :3] -= block[:, :3].min(0) - np.float32(0.001)     # down to the first cells
    pos = shuffled(block)
    n = len(pos)
    stray = np.array([[0.02, 0.02, 0.02, 0.0]], np.float32)
    stray[0, axis] = away
    clean = run(gsph, p, pos)
    got = run(gsph, p, np.concatenate([pos, stray]))
    assert got["tasks"] > 0 and clean["tasks"] > 0
    # per source particle, without the stray one
    keep = got["perm"] < n
    back = np.empty(n, np.int64)
    back[got["perm"][keep]] = np.flatnonzero(keep)
    rows = back[clean["perm"]]                                   # in the clean run's order
    rho, _ = oracle.density(clean["POSITION"], clean["KEY"], clean["CELL_START"], p)
    gpu = 1.0 / got["POSITION"][rows, 3].astype(np.float64)
    assert np.max(np.abs(gpu - rho) / rho) <= RHO_TOL
    force, mag = oracle.force(clean["POSITION"], clean["EVAL_VELOCITY"], clean["KEY"],
                              clean["CELL_START"], p, with_mag=True)
    fn = np.linalg.norm(force, axis=1)
    # (the stray run's own densities and pressures differ by their rounding)
    bound = FORCE_TOL * np.maximum(fn, np.sqrt(np.mean(fn ** 2))) + FORCE_SUM_TOL * mag
    dev = np.linalg.norm(got["ACCELERATION"][rows, :3].astype(np.float64) - force, axis=1)
    assert np.all(dev <= bound), (dev / bound).max()
    assert np.isfinite(got["ACCELERATION"]).all()
