"""gsph_step_host_async overlaps its copies with the first and last frame's
passes (velocities go up while the positions are sorted and the density pass
runs; past the small-scene builds the state goes back in parts of the force
pass). Its results are those of frames on resident state, bit for bit, for
every way the frames are launched, for scenes with small cells, cells of the
block-level sort, both paths side by side, and sizes that divide by nothing."""
import numpy as np
import pytest

from gpu_helpers import dam_scene, dense_scene, shuffled

pytestmark = pytest.mark.gpu


def mixed(gsph, n_side=18, loose=3001):
    """A dense block (SMS, cells past 32 particles) in a sparse cloud (TRA)."""
    _, p, dense = dense_scene(gsph, n_side=n_side)
    rng = np.random.default_rng(3)
    cloud = np.zeros((loose, 4), np.float32)
    cloud[:, :3] = rng.uniform(0.2, 0.4, (len(cloud), 3))
    return None, p, np.concatenate([dense, cloud])


SCENES = {
    "one": lambda g: (None, dam_scene(g, n_side=4)[1], dam_scene(g, n_side=4)[2][:1]),
    "odd": lambda g: (None, *[dam_scene(g, n_side=13)[k] for k in (1, 2)]),
    "past the small builds": lambda g: dam_scene(g, n_side=52, box=(1.2, 1.2, 1.2)),
    "mixed": mixed,
    "mixed, in parts": lambda g: mixed(g, n_side=52, loose=9001),
}


@pytest.mark.parametrize("graph,frames", [(0, 1), (0, 3), (2, 1), (2, 3)])
@pytest.mark.parametrize("name", sorted(SCENES))
def test_overlapped_copies_change_no_bits(gsph, cuda_device, name, graph, frames):
    import torch
    _, p, pos = SCENES[name](gsph)
    pos = shuffled(pos)
    vel = np.zeros_like(pos)
    vel[:, :3] = np.random.default_rng(1).normal(0.0, 0.2, (len(pos), 3))
    fields = (gsph.FIELD_POSITION, gsph.FIELD_VELOCITY, gsph.FIELD_EVAL_VELOCITY)
    calls = 3
    with gsph.HybridSystem(params=p, positions=pos, velocities=vel) as h:
        h.set_graph_mode(graph)
        host = [torch.empty((h.n, 4), dtype=torch.float32, pin_memory=True) for _ in range(3)]
        for t, a in zip(host, (pos, vel, vel)):
            t.numpy()[:] = a
        for _ in range(calls):
            h.step_host_async(frames, *(t.data_ptr() for t in host))
        h.sync()
        got = [t.numpy().copy() for t in host] + [h.copy_out(gsph.FIELD_ACCELERATION)]
        dev = [h.copy_out(f) for f in fields]
    with gsph.HybridSystem(params=p, positions=pos, velocities=vel) as r:
        r.copy_in(gsph.FIELD_EVAL_VELOCITY, vel)
        r.step(calls * frames)
        ref = [r.copy_out(f) for f in fields] + [r.copy_out(gsph.FIELD_ACCELERATION)]
    for a, b in zip(got + dev, ref + ref[:3]):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
