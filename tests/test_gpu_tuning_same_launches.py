"""Small scenes' TRA kernels ignore the TRA block counts, so tunings that differ
in nothing else launch the same: the autotuner tries the first of them and does
not let noise choose among the rest."""
import pytest

from gpu_helpers import dam_scene, shuffled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_side", [12, 30])
def test_equal_launches_are_not_told_apart_by_noise(gsph, cuda_device, n_side):
    _, p, pos = dam_scene(gsph, n_side=n_side, box=(0.9, 0.5, 0.5))
    candidates = []
    for density in (5, 6, 4, 3, 2):
        for force in (3, 4, 2, 1):
            t = gsph.tuning_default()
            t.ctas_density_tra, t.ctas_force_tra = density, force
            candidates.append(t)
    with gsph.HybridSystem(params=p, positions=shuffled(pos)) as h:
        for _ in range(4):
            best, ms = h.autotune(frames_per_trial=1, candidates=candidates)
            assert ms > 0
            assert best.as_dict() == candidates[0].as_dict()
            assert h.get_tuning().as_dict() == best.as_dict()
