"""SMS passes at the sizes where a cell's particles divide unevenly into tasks
(32 particles), clusters (16), candidate pairs, runs of 64 tested candidates
and batches of 128 staged ones: density and force against the FP64 oracle with
the parity bounds (density 1e-5; force 1e-4 of |F| plus 64 u times the sum of
the pair-term magnitudes), and the same bits for a scene alone, in a batch
after another scene, and with blocks of 4 warps."""
import numpy as np
import pytest

from gpu_helpers import dense_scene

pytestmark = pytest.mark.gpu

RHO_TOL, FORCE_TOL, SUM_TOL = 1e-5, 1e-4, 64 * 2.0 ** -24


def clumps(p, n, seed):
    """n particles inside one cell, n around a corner of eight cells, 2n over
    a row of cells at the grid's lower x edge: every count of the n range."""
    rng = np.random.default_rng(seed)
    h = float(p.kernel)
    parts = [(np.array([4, 4, 4]) + rng.uniform(0.02, 0.98, (n, 3))) * h,
             (np.array([9, 6, 8]) + rng.uniform(-0.6, 0.6, (n, 3))) * h,
             np.array([0.0, 9 * h, 3 * h]) + rng.uniform(0.02, 0.98, (2 * n, 3)) *
             np.array([3 * h, h, h])]
    pos = np.zeros((sum(map(len, parts)), 4), np.float32)
    pos[:, :3] = np.concatenate(parts)
    vel = np.zeros_like(pos)
    vel[:, :3] = rng.normal(3.0, 0.05, (len(pos), 3))   # a common motion, small differences
    order = rng.permutation(len(pos))
    return pos[order].copy(), vel[order].copy()


def evaluate(gsph, sysm, ev, artificial):
    if artificial:
        sysm.set_viscosity_model(gsph.VISCOSITY_ARTIFICIAL, 0.02, 20.0)
    sysm.copy_in(gsph.FIELD_EVAL_VELOCITY, ev)
    sysm.arrange()
    sysm.density()
    sysm.force()
    return [sysm.copy_out(f) for f in (gsph.FIELD_POSITION, gsph.FIELD_EVAL_VELOCITY,
                                       gsph.FIELD_ACCELERATION)]


@pytest.mark.parametrize("artificial", [False, True])
@pytest.mark.parametrize("n", [15, 16, 17, 31, 32, 33, 47, 49, 63, 65, 130, 1023, 1030])
def test_clusters_vs_fp64(gsph, oracle, cuda_device, n, artificial):
    _, p, _ = dense_scene(gsph, n_side=4)
    pos, vel = clumps(p, n, n)
    with gsph.HybridSystem(params=p, positions=pos, velocities=vel) as sysm:
        spos, sev, acc = evaluate(gsph, sysm, vel, artificial)
        assert sysm.copy_out(gsph.FIELD_SPLIT)[1] > 0
        ks, cs = sysm.copy_out(gsph.FIELD_KEY), sysm.copy_out(gsph.FIELD_CELL_START)
        t = sysm.get_tuning()
    rho, _ = oracle.density(spos, ks, cs, p)
    assert (np.abs(1.0 / spos[:, 3].astype(np.float64) - rho) / rho).max() <= RHO_TOL
    if artificial:
        ref, mag = oracle.force(spos, sev, ks, cs, p, with_mag=True, artificial=(0.02, 20.0))
    else:
        ref, mag = oracle.force(spos, sev, ks, cs, p, with_mag=True)
    fn = np.linalg.norm(ref, axis=1)
    bound = FORCE_TOL * np.maximum(fn, 1e-3 * np.sqrt(np.mean(fn ** 2))) + SUM_TOL * mag
    dev = np.linalg.norm(acc[:, :3].astype(np.float64) - ref, axis=1)
    assert np.all(dev <= bound), (dev / bound).max()

    other, ovel = clumps(p, 40, 99)
    with gsph.Batch([(p, other, ovel), (p, pos, vel)]) as b:
        both = evaluate(gsph, b, np.concatenate([ovel, vel]), artificial)
        got = [a[len(other):] for a in both]
    with gsph.HybridSystem(params=p, positions=pos, velocities=vel) as sysm:
        t.warps_per_block = 4
        sysm.set_tuning(t)
        half = evaluate(gsph, sysm, vel, artificial)
    for a, x, y in zip((spos, sev, acc), got, half):
        assert np.array_equal(a.view(np.uint32), x.view(np.uint32))
        assert np.array_equal(a.view(np.uint32), y.view(np.uint32))
