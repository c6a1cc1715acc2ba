"""A batch whose scenes are replaced by one without particles reports an empty
grid after its next frame: the scatter, which publishes the number of large
cells, is not launched then."""
import numpy as np
import pytest

from gpu_helpers import dense_scene

pytestmark = pytest.mark.gpu


def test_an_emptied_batch_reports_no_cells(gsph, cuda_device):
    _, p, pos = dense_scene(gsph, n_side=14)
    empty = (p, np.zeros((0, 4), np.float32))
    with gsph.Batch([(p, pos)]) as b:
        b.step(1)
        info = b.info()
        assert info.big_cells > 0 and info.occupied_cells > 0 and info.sms_tasks > 0
        b.repack([], [empty])
        b.step(1)
        info = b.info()
        assert (info.n_particles, info.occupied_cells, info.big_cells, info.sms_tasks,
                info.tra_particles) == (0, 0, 0, 0, 0)
        b.repack([], [(p, pos)])   # and full again
        b.step(1)
        got = b.copy_out(gsph.FIELD_POSITION)
    with gsph.HybridSystem(params=p, positions=pos) as h:
        h.step(1)
        assert np.array_equal(got.view(np.uint32), h.copy_out(gsph.FIELD_POSITION).view(np.uint32))
