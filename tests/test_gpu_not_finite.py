"""A particle without neighbours whose evaluated velocity is not finite takes no
force, in the smallest scenes' force pass (four lanes per particle, rounds as
long as the busiest particle of the warp's) as in the general one, and changes
no other particle."""
import numpy as np
import pytest

from gpu_helpers import dam_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("artificial", [False, True])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_a_lone_particle_that_is_not_finite(gsph, cuda_device, value, artificial):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    _, p, filler = dam_scene(gsph, n_side=int(np.ceil((41 * sms * 32) ** (1 / 3))),
                             box=(1.2, 1.2, 1.2))
    assert len(filler) > 40 * sms * 32
    _, _, block = dam_scene(gsph, n_side=4, box=(1.2, 1.2, 1.2))
    lone = np.array([[0.03, 0.03, 0.012, 0.0]], np.float32)   # first in the sorted order
    pos = np.concatenate([block, lone])

    def force(h):
        if artificial:
            h.set_viscosity_model(gsph.VISCOSITY_ARTIFICIAL, 0.02, 20.0)
        ev = h.copy_out(gsph.FIELD_EVAL_VELOCITY)
        ev[len(block), :3] = value
        h.copy_in(gsph.FIELD_EVAL_VELOCITY, ev)
        h.arrange()
        h.density()
        h.force()
        assert h.copy_out(gsph.FIELD_PERMUTATION)[0] == len(block)
        assert h.copy_out(gsph.FIELD_NEIGHBOR_COUNT)[0] == 0
        return h.copy_out(gsph.FIELD_ACCELERATION)[:len(pos)]

    with gsph.HybridSystem(params=p, positions=pos) as h:
        alone = force(h)
    with gsph.Batch([(p, pos), (p, filler)]) as b:
        both = force(b)
    assert np.isfinite(both).all() and np.any(both[1:] != 0)
    assert np.array_equal(alone.view(np.uint32), both.view(np.uint32))
