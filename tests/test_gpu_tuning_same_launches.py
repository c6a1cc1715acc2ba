"""Small scenes' TRA kernels ignore the TRA block counts, so tunings that differ
in nothing else launch the same: the autotuner tries the first of them and does
not let noise choose among the rest. So do the SMS force pass's counts beyond
what an SM holds."""
import pytest

from gpu_helpers import dam_scene, dense_scene, shuffled

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


@pytest.mark.parametrize("warps,counts", [(8, (4, 3)), (4, (7, 8, 6))])
def test_sms_force_counts_past_the_resident_ones_launch_the_same(gsph, cuda_device, warps,
                                                                 counts):
    _, p, pos = dense_scene(gsph, n_side=40)
    candidates = []
    for count in counts:
        t = gsph.tuning_default()
        t.warps_per_block, t.ctas_force_sms = warps, count
        candidates.append(t)
    state = []
    with gsph.HybridSystem(params=p, positions=shuffled(pos)) as h:
        for _ in range(8):
            best, _ = h.autotune(frames_per_trial=1, candidates=candidates)
            assert best.as_dict() == candidates[0].as_dict()
    for t in candidates:
        with gsph.HybridSystem(params=p, positions=shuffled(pos)) as h:
            h.set_tuning(t)
            h.step(2)
            state.append(h.copy_out(gsph.FIELD_POSITION))
    for other in state[1:]:
        assert (other == state[0]).all()
