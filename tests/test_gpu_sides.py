"""The two streams of a frame change over once the TRA passes fill the GPU for
long (more than 128 units of 32 particles per SM). A scene below that size gives
the same bits alone and in a batch above it, launched kernel by kernel and from
graphs, and a large mixed scene the same bits frame by frame and stage by
stage."""
import numpy as np
import pytest

from gpu_helpers import dense_scene, shuffled

pytestmark = pytest.mark.gpu


def mixed(gsph, n_side, loose, seed):
    """A dense block (SMS) in a sparse cloud (TRA)."""
    _, p, dense = dense_scene(gsph, n_side=n_side)
    cloud = np.zeros((loose, 4), np.float32)
    cloud[:, :3] = np.random.default_rng(seed).uniform(0.05, 0.45, (loose, 3))
    return p, shuffled(np.concatenate([dense, cloud]), seed=seed)


def fields(gsph):
    return (gsph.FIELD_POSITION, gsph.FIELD_VELOCITY, gsph.FIELD_EVAL_VELOCITY,
            gsph.FIELD_KEY)


def same(a, b):
    return all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(a, b))


def test_scenes_below_the_line_in_a_batch_above_it(gsph, cuda_device):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    scenes = [mixed(gsph, 20, 30001, 1), mixed(gsph, 5, 40007, 2), mixed(gsph, 12, 9, 3)]
    _, p, block = dense_scene(gsph, n_side=88)
    scenes.append((p, block))
    assert sum(len(pos) for _, pos in scenes) > sms * 128 * 32
    alone = []
    for q, pos in scenes[:3]:
        with gsph.HybridSystem(params=q, positions=pos) as h:
            h.step(3)
            alone.append([h.copy_out(f) for f in fields(gsph)])
    for graph in (0, 3):
        with gsph.Batch(scenes) as b:
            b.set_graph_mode(graph)
            b.step(3)
            assert b.info().sms_tasks > 0
            for k in range(3):
                assert same([b.copy_out_scene(k, f) for f in fields(gsph)], alone[k])


def test_a_large_mixed_scene_frame_by_frame_and_by_stages(gsph, cuda_device):
    p, pos = mixed(gsph, 80, 200003, 4)
    got = []
    for how in ("frames", "graph", "stages"):
        with gsph.HybridSystem(params=p, positions=pos) as h:
            h.set_graph_mode(2 if how == "graph" else 0)
            if how == "stages":
                for _ in range(2):
                    h.arrange()
                    h.density()
                    h.force()
                    h.advance()
            else:
                h.step(2)
            got.append([h.copy_out(f) for f in fields(gsph)])
    assert same(got[0], got[1]) and same(got[0], got[2])
