"""gsph_density and gsph_force called again on the same grid compute anew from
the state as it is, whichever kernels the scene's size selects: after the
evaluated velocities have changed, a second force call gives what a fresh
handle gives, and a second density call restores a pressure that the caller
overwrote. The general TRA kernels (past the small-scene builds) and SMS scenes
with more clusters than resident warps take their work from queues that the
first call has used up."""
import numpy as np
import pytest

from gpu_helpers import dam_scene, dense_scene, shuffled

pytestmark = pytest.mark.gpu


def mixed(gsph, n_side, loose, seed):
    """A dense block (SMS) in a sparse cloud (TRA)."""
    _, p, dense = dense_scene(gsph, n_side=n_side)
    cloud = np.zeros((loose, 4), np.float32)
    cloud[:, :3] = np.random.default_rng(seed).uniform(0.05, 0.45, (loose, 3))
    return p, np.concatenate([dense, cloud])


def scene(gsph, name, sms):
    if name == "smallest":
        p, pos = dam_scene(gsph, n_side=12)[1:]
    elif name == "small":
        p, pos = dam_scene(gsph, n_side=40, box=(1.0, 1.0, 1.0))[1:]
    elif name == "general":
        side = int(np.ceil((41 * sms * 32) ** (1 / 3)))
        p, pos = dam_scene(gsph, n_side=side, box=(1.2, 1.2, 1.2))[1:]
        assert len(pos) > 40 * sms * 32
    elif name == "mixed":
        p, pos = mixed(gsph, 16, 4001, 1)
    else:   # more clusters of 16 than the SMs hold warps of the SMS passes
        side = int(np.ceil((40 * sms * 16) ** (1 / 3)))
        p, pos = mixed(gsph, side, 41 * sms * 32, 2)
    return p, shuffled(pos)


@pytest.mark.parametrize("name", ["smallest", "small", "general", "mixed", "mixed, queued"])
def test_a_repeated_stage_computes_anew(gsph, cuda_device, name):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    p, pos = scene(gsph, name, sms)

    def prepared():
        h = gsph.HybridSystem(params=p, positions=pos)
        h.arrange()
        h.density()
        return h

    def changed(ev):
        out = ev.copy()
        out[:, :3] = np.random.default_rng(5).normal(0.0, 0.5, (len(ev), 3))
        return out

    with prepared() as h:
        h.force()
        before = h.copy_out(gsph.FIELD_ACCELERATION)
        ev = h.copy_out(gsph.FIELD_EVAL_VELOCITY)
        h.copy_in(gsph.FIELD_EVAL_VELOCITY, changed(ev))
        h.force()
        again = h.copy_out(gsph.FIELD_ACCELERATION)
        overwritten = ev.copy()
        overwritten[:, 3] = -1.0
        h.copy_in(gsph.FIELD_EVAL_VELOCITY, overwritten)
        h.density()
        restored = h.copy_out(gsph.FIELD_EVAL_VELOCITY)
        h.force()
        last = h.copy_out(gsph.FIELD_ACCELERATION)
    with prepared() as h:
        ev_f = h.copy_out(gsph.FIELD_EVAL_VELOCITY)
        h.copy_in(gsph.FIELD_EVAL_VELOCITY, changed(ev_f))
        h.force()
        fresh = h.copy_out(gsph.FIELD_ACCELERATION)
    assert np.array_equal(ev, ev_f)
    assert not np.array_equal(before, fresh)
    assert np.array_equal(again, fresh)
    assert np.array_equal(restored, ev)
    assert np.array_equal(last, before)


def test_a_captured_force_call_can_be_replayed(gsph, cuda_device):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    p, pos = scene(gsph, "mixed, queued", sms)
    with gsph.HybridSystem(params=p, positions=pos) as h:
        h.arrange()
        h.density()
        ev = h.copy_out(gsph.FIELD_EVAL_VELOCITY)
        stream = torch.cuda.ExternalStream(h.stream())
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(stream):
            graph.capture_begin(capture_error_mode="thread_local")
            h.force()
            graph.capture_end()
            graph.replay()
        first = h.copy_out(gsph.FIELD_ACCELERATION)
        ev[:, :3] = np.random.default_rng(5).normal(0.0, 0.5, (len(ev), 3))
        h.copy_in(gsph.FIELD_EVAL_VELOCITY, ev)
        with torch.cuda.stream(stream):
            graph.replay()
        second = h.copy_out(gsph.FIELD_ACCELERATION)
        h.force()
        plain = h.copy_out(gsph.FIELD_ACCELERATION)
    assert not np.array_equal(first, second)
    # (the captured launch walks the masks, the plain one after a copy-in scans)
    assert np.allclose(second, plain, rtol=1e-3, atol=1e-3 * np.abs(plain).max())


def test_captured_stages_with_their_arrange_can_be_replayed(gsph, cuda_device):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    p, pos = scene(gsph, "mixed, queued", sms)
    fields = (gsph.FIELD_POSITION, gsph.FIELD_EVAL_VELOCITY, gsph.FIELD_ACCELERATION)
    with gsph.HybridSystem(params=p, positions=pos) as h:
        h.arrange()
        h.density()
        h.force()
        ref = [h.copy_out(f) for f in fields]
    with gsph.HybridSystem(params=p, positions=pos) as h:
        stream = torch.cuda.ExternalStream(h.stream())
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(stream):
            graph.capture_begin(capture_error_mode="thread_local")
            h.arrange()
            h.density()
            h.force()
            graph.capture_end()
            for _ in range(2):
                graph.replay()
        got = [h.copy_out(f) for f in fields]
        h.density()   # and a plain call after them
        h.force()
        again = [h.copy_out(f) for f in fields]
    for a, b, c in zip(ref, got, again):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
        assert np.array_equal(a.view(np.uint32), c.view(np.uint32))
