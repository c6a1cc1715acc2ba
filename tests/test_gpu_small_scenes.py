"""The TRA passes choose among builds by the number of particles: density with
a work unit's rows spread over nine or three warps or walked by one, force with
four lanes per particle, or with four or two neighbours in flight. A scene gives the same bits whichever runs:
alone (a small-scene build) and in a batch large enough for the general ones.
Sizes sit around the rules' lines (units per SM times 152 SMs times 32
particles); the crowded scenes have rows of more than 32 candidates (no mask)
and more than 12 interacting ones (past the terms kept in shared memory), and
particles with more than 64 neighbours (past the four lanes' list)."""
import numpy as np
import pytest

from gpu_helpers import dam_scene, shuffled

pytestmark = pytest.mark.gpu


def state(gsph, sysm, all_tra):
    if all_tra:   # no cell takes the SMS path, however crowded
        t = sysm.get_tuning()
        t.sparse_total = t.sparse_self = 1 << 30
        sysm.set_tuning(t)
    sysm.step(2)
    sysm.arrange()
    sysm.density()
    count = sysm.copy_out(gsph.FIELD_NEIGHBOR_COUNT)
    sysm.force()
    return [sysm.copy_out(f) for f in (gsph.FIELD_POSITION, gsph.FIELD_VELOCITY,
                                       gsph.FIELD_EVAL_VELOCITY, gsph.FIELD_ACCELERATION)] + [
        count]


CASES = {   # particles, positions pulled together by
    "one": (1, 1.0), "quad+1": (9, 1.0), "unit-1": (31, 1.0), "unit+1": (33, 1.0), "odd": (1501, 1.0),
    "row-per-warp": (24320, 1.0), "three-rows": (24321, 1.0), "force-line": (82689, 1.0),
    "row-per-warp again": (43777, 1.0), "three-rows again": (53505, 1.0),
    "three-rows end": (87552, 1.0), "general density": (87553, 1.0),
    "force-small end": (102144, 1.0), "force general": (102145, 1.0),
    "force-small again": (165377, 1.0), "force-small again end": (194560, 1.0),
    "crowded": (2000, 0.6), "very crowded": (2000, 0.2), "crowded, three rows": (30000, 0.3),
}


@pytest.mark.parametrize("artificial", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_small_scene_builds_give_the_same_bits(gsph, cuda_device, name, artificial):
    n, squeeze = CASES[name]
    side = int(np.ceil(n ** (1 / 3)))
    box = (1.6, 1.2, 1.0)
    _, p, pos = dam_scene(gsph, n_side=side, box=box)
    pos = shuffled(pos)[:n]
    if squeeze < 1.0:
        away = pos[:, :3] - pos[:, :3].mean(0)       # densest in the middle
        r = np.linalg.norm(away, axis=1, keepdims=True)
        pos[:, :3] -= away * (1 - np.float32(squeeze)) * (1 - r / r.max())
    _, _, filler = dam_scene(gsph, n_side=54, box=box, seed=3)     # 157,464 particles
    with gsph.HybridSystem(params=p, positions=pos) as a:
        if artificial:
            a.set_viscosity_model(gsph.VISCOSITY_ARTIFICIAL, 0.02, 20.0)
        alone = state(gsph, a, squeeze < 1.0)
    with gsph.Batch([(p, pos), (p, filler)]) as b:
        if artificial:
            b.set_viscosity_model(gsph.VISCOSITY_ARTIFICIAL, 0.02, 20.0)
        both = state(gsph, b, squeeze < 1.0)
    if name == "very crowded":
        assert alone[4].min() < 0 and alone[4].max() > 0   # rows past the mask, and within it
    for x, y in zip(alone, both):
        assert np.array_equal(x.view(np.uint32), y[:n].view(np.uint32))
