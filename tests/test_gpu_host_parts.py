"""gsph_step_host_async on scenes large enough that the last force pass runs in
parts, each part's rows on their way back while the next is computed (more than
76 units of 32 particles per SM): the results are those of frames on resident
state, bit for bit, for both viscosity models, both block shapes, a batch, TRA
particles alone and beside SMS cells, and host arrays that are not pinned."""
import numpy as np
import pytest

from gpu_helpers import dam_scene, dense_scene, shuffled

pytestmark = pytest.mark.gpu

PARTS = 76


def sparse(gsph, count, seed):
    side = int(np.ceil(count ** (1 / 3)))
    _, p, pos = dam_scene(gsph, n_side=side, box=(1.6, 1.6, 1.6), seed=seed)
    return p, shuffled(pos, seed=seed)


def mixed(gsph, count, seed):
    """A dense block (SMS) in a sparse cloud (TRA)."""
    _, p, dense = dense_scene(gsph, n_side=24, seed=seed)
    cloud = np.zeros((count, 4), np.float32)
    cloud[:, :3] = np.random.default_rng(seed).uniform(0.05, 0.45, (count, 3))
    return p, shuffled(np.concatenate([dense, cloud]), seed=seed)


CASES = {   # scene, scenes in the batch (0: a single scene), artificial, warps, frames, pinned
    "sparse": (sparse, 0, False, 8, 1, True),
    "sparse, frames": (sparse, 0, False, 8, 3, True),
    "mixed": (mixed, 0, False, 8, 2, True),
    "artificial": (sparse, 0, True, 8, 1, True),
    "artificial, mixed": (mixed, 0, True, 8, 1, True),
    "four warps": (sparse, 0, False, 4, 1, True),
    "four warps, artificial, mixed": (mixed, 0, True, 4, 2, True),
    "batch": (sparse, 3, False, 8, 2, True),
    "batch, four warps, artificial": (sparse, 2, True, 4, 1, True),
    "not pinned": (sparse, 0, False, 8, 2, False),
    "not pinned, mixed": (mixed, 0, False, 8, 1, False),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_parts_change_no_bits(gsph, cuda_device, name):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    build, scenes, artificial, warps, frames, pinned = CASES[name]
    count = (PARTS + 1) * sms * 32 // max(scenes, 1) + 77
    made = [build(gsph, count, seed) for seed in range(max(scenes, 1))]
    rng = np.random.default_rng(1)
    n = sum(len(pos) for _, pos in made)
    assert n > PARTS * sms * 32
    pos = np.concatenate([q for _, q in made])
    vel = np.zeros_like(pos)
    vel[:, :3] = rng.normal(0.0, 0.2, (n, 3))
    fields = (gsph.FIELD_POSITION, gsph.FIELD_VELOCITY, gsph.FIELD_EVAL_VELOCITY)

    def handle():
        h = (gsph.Batch(made) if scenes
             else gsph.HybridSystem(params=made[0][0], positions=pos))
        h.copy_in(gsph.FIELD_VELOCITY, vel)
        h.copy_in(gsph.FIELD_EVAL_VELOCITY, vel)
        if artificial:
            h.set_viscosity_model(gsph.VISCOSITY_ARTIFICIAL, 0.02, 20.0)
        if warps != 8:
            t = h.get_tuning()
            t.warps_per_block = warps
            h.set_tuning(t)
        return h

    calls = 2
    with handle() as h:
        host = [torch.empty((n, 4), dtype=torch.float32, pin_memory=pinned) for _ in range(3)]
        for t, a in zip(host, (pos, vel, vel)):
            t.numpy()[:] = a
        for _ in range(calls):
            h.step_host_async(frames, *(t.data_ptr() for t in host))
        h.sync()
        got = [t.numpy().copy() for t in host] + [h.copy_out(gsph.FIELD_ACCELERATION)]
        got += [h.copy_out(f) for f in fields]
    with handle() as r:
        r.step(calls * frames)
        if build is mixed:
            assert r.info().sms_tasks > 0
        ref = [r.copy_out(f) for f in fields] + [r.copy_out(gsph.FIELD_ACCELERATION)]
    for a, b in zip(got, ref + ref[:3]):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
