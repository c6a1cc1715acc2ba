"""The general builds of the TRA passes: blocks of 8 and of 4 warps, the density
pass with and without the prefetch of its rows' cell offsets (cell arrays above
64 MB), and for one scene and several. The same fluid gives the same bits per
particle in all of them. Every scene is past the small-scene builds, which
ignore the block shape and do not prefetch, by the rule's own lines."""
import re
from pathlib import Path

import numpy as np
import pytest

from gpu_helpers import dam_scene, shuffled

pytestmark = pytest.mark.gpu

SOURCE = (Path(__file__).resolve().parent.parent / "fast-general-gpu-sph-framework_gb300" /
          "csrc" / "physics.cu")
LINES = [int(v) for v in re.findall(r"\bk(?:Rows|ForceQuad|ForceSmall)\w* = (\d+)",
                                    SOURCE.read_text())]
SMALL = (1.0, 1.0, 1.0)       # 50^3 cells, 1 MB of cell offsets and slab words
LARGE = (5.12, 5.12, 3.2)     # 10,485,760 cells, 84 MB


@pytest.fixture(scope="module")
def fluid(gsph, cuda_device):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    need = max(LINES) * sms * 32
    side = int(np.ceil((need + 1) ** (1 / 3)))
    params, made = {}, {}
    for name, box in (("small", SMALL), ("large", LARGE)):
        _, params[name], made[name] = dam_scene(gsph, n_side=side, box=box)
    assert np.array_equal(made["small"], made["large"]) and len(made["small"]) > need
    cells = {k: int(np.prod(np.asarray(p.grid_size, np.int64))) for k, p in params.items()}
    assert cells["small"] * 8 < 64 << 20 < cells["large"] * 8
    pos = shuffled(made["small"], seed=4)
    vel = np.zeros_like(pos)
    vel[:, :3] = np.random.default_rng(6).normal(0.0, 0.3, (len(pos), 3))
    return params, pos, vel


def run(gsph, fluid, box, scenes, warps, artificial):
    """Per source particle of the first scene: density, pressure, force, and the
    state two frames later."""
    params, pos, vel = fluid
    p, n = params[box], len(pos)
    with (gsph.Batch([(p, pos, vel)] * scenes) if scenes > 1 else
          gsph.HybridSystem(params=p, positions=pos, velocities=vel)) as h:
        t = h.get_tuning()
        t.warps_per_block = warps
        h.set_tuning(t)
        if artificial:
            h.set_viscosity_model(gsph.VISCOSITY_ARTIFICIAL, 0.02, 20.0)
        h.arrange()
        h.copy_in(gsph.FIELD_EVAL_VELOCITY, h.copy_out(gsph.FIELD_VELOCITY))
        h.density()
        assert h.info().sms_tasks == 0
        h.force()
        perm = h.copy_out(gsph.FIELD_PERMUTATION)
        first = [h.copy_out(f) for f in (gsph.FIELD_POSITION, gsph.FIELD_EVAL_VELOCITY,
                                         gsph.FIELD_ACCELERATION)]
        first.append(h.copy_out(gsph.FIELD_NEIGHBOR_COUNT))
        out = []
        for a in first:
            by_source = np.empty_like(a)
            by_source[perm] = a
            out.append(by_source[:n])
        h.step(2)
        out += [h.copy_out(f)[:n] for f in (gsph.FIELD_POSITION, gsph.FIELD_VELOCITY,
                                            gsph.FIELD_EVAL_VELOCITY)]
    return out


@pytest.fixture(scope="module")
def reference(gsph, fluid):
    return {a: run(gsph, fluid, "small", 1, 8, a) for a in (False, True)}


@pytest.mark.parametrize("artificial", [False, True])
@pytest.mark.parametrize("warps", [8, 4])
@pytest.mark.parametrize("scenes", [1, 2])
@pytest.mark.parametrize("box", ["small", "large"])
def test_the_general_builds_agree(gsph, fluid, reference, box, scenes, warps, artificial):
    got = run(gsph, fluid, box, scenes, warps, artificial)
    for k, (x, y) in enumerate(zip(reference[artificial], got)):
        # the order after a frame follows the cells' numbers, the same in both boxes
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), k


def test_the_reference_matches_fp64(gsph, oracle, fluid):
    params, pos, vel = fluid
    with gsph.HybridSystem(params=params["small"], positions=pos, velocities=vel) as h:
        h.arrange()
        h.density()
        q = h.copy_out(gsph.FIELD_POSITION)
        key, start = h.copy_out(gsph.FIELD_KEY), h.copy_out(gsph.FIELD_CELL_START)
    rho, _ = oracle.density(q, key, start, params["small"])
    assert np.max(np.abs(1.0 / q[:, 3].astype(np.float64) - rho) / rho) <= 1e-5
