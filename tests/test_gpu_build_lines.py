"""The small-scene builds of the TRA passes against the general ones, at every
line of the rule that chooses them. The lines (units of 32 particles per SM) are
read from the dispatch itself and the sizes follow from the GPU's SM count, so the
cases stay on the lines whatever either is. A scene alone runs the build of its
size; in a batch whose filler puts it above every line it runs the general
builds; the bits are the same. Crowded scenes have particles with a row of more
than 32 candidates (no masks) beside others (with masks)."""
import re
from pathlib import Path

import numpy as np
import pytest

from gpu_helpers import dam_scene, shuffled

pytestmark = pytest.mark.gpu

SOURCE = (Path(__file__).resolve().parent.parent / "fast-general-gpu-sph-framework_gb300" /
          "csrc" / "physics.cu")
LINES = {k: int(v) for k, v in
         re.findall(r"\b(kRows\w+|kForce(?:Quad|Small)\w+) = (\d+)", SOURCE.read_text())}
NAMES = ("kRowsMax1", "kRowsAgain1", "kRowsAgainMax1", "kRowsMax3", "kForceQuadMax",
         "kForceSmallMax", "kForceSmallAgain", "kForceSmallAgainMax")
BOX = (1.6, 1.2, 1.0)


@pytest.fixture(scope="module")
def sms(cuda_device):
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.fixture(scope="module")
def filler(gsph, sms):
    """Particles that by themselves are past every line."""
    count = (max(LINES.values()) + 1) * sms * 32
    _, p, pos = dam_scene(gsph, n_side=int(np.ceil(count ** (1 / 3))), box=BOX, seed=3)
    assert len(pos) > max(LINES.values()) * sms * 32
    return p, pos


def state(gsph, h, n, artificial):
    t = h.get_tuning()
    t.sparse_total = t.sparse_self = 1 << 30   # all TRA, however crowded
    h.set_tuning(t)
    if artificial:
        h.set_viscosity_model(gsph.VISCOSITY_ARTIFICIAL, 0.02, 20.0)
    h.step(2)
    h.arrange()
    h.density()
    count = h.copy_out(gsph.FIELD_NEIGHBOR_COUNT)[:n]
    h.force()
    return count, [h.copy_out(f)[:n] for f in
                   (gsph.FIELD_POSITION, gsph.FIELD_VELOCITY, gsph.FIELD_EVAL_VELOCITY,
                    gsph.FIELD_ACCELERATION)]


def compare(gsph, filler, pos, artificial):
    p, fill = filler
    n = len(pos)
    with gsph.HybridSystem(params=p, positions=pos) as a:
        count, alone = state(gsph, a, n, artificial)
    with gsph.Batch([(p, pos), (p, fill)]) as b:
        count_b, both = state(gsph, b, n, artificial)
    assert np.array_equal(count, count_b)
    for x, y in zip(alone, both):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
    return count


@pytest.mark.parametrize("artificial", [False, True])
@pytest.mark.parametrize("beyond", [0, 1])
@pytest.mark.parametrize("line", NAMES)
def test_the_same_bits_on_both_sides_of_each_line(gsph, sms, filler, line, beyond, artificial):
    assert sorted(LINES) == sorted(NAMES)
    n = LINES[line] * sms * 32 + beyond
    _, _, pos = dam_scene(gsph, n_side=int(np.ceil(n ** (1 / 3))), box=BOX)
    compare(gsph, filler, shuffled(pos)[:n], artificial)


def crowded(gsph, n, squeeze):
    """A block pulled together towards its middle."""
    _, _, pos = dam_scene(gsph, n_side=int(np.ceil(n ** (1 / 3))), box=BOX)
    pos = shuffled(pos)[:n]
    away = pos[:, :3] - pos[:, :3].mean(0)
    r = np.linalg.norm(away, axis=1, keepdims=True)
    pos[:, :3] -= away * (1 - np.float32(squeeze)) * (1 - r / r.max())
    return pos


@pytest.mark.parametrize("artificial", [False, True])
@pytest.mark.parametrize("units", ["kForceQuadMax", "kRowsMax1", "kRowsAgainMax1", "kRowsMax3",
                                   "kForceSmallMax", "kForceSmallAgainMax"])
def test_the_same_bits_in_crowded_scenes(gsph, sms, filler, units, artificial):
    count = compare(gsph, filler, crowded(gsph, LINES[units] * sms * 32, 0.3), artificial)
    assert count.min() == -1 and count.max() > 32
