"""The cell scan in its three forms: the earlier tiles' counts added up by each
block, the earlier tiles' sums, and the sums scanned by one block first (above
16.8M cells). Grids on both sides of both lines: offsets, order, performance
model, split and tasks equal the oracle's, and the numbers of occupied and of
large cells a direct count."""
import re
from pathlib import Path

import numpy as np
import pytest

from gpu_helpers import dam_scene

pytestmark = pytest.mark.gpu

HEADER = (Path(__file__).resolve().parent.parent / "fast-general-gpu-sph-framework_gb300" /
          "csrc" / "gsph_internal.h")
H = 0.02


def constant(name):
    return int(re.search(rf"\b{name} = (\d+);", HEADER.read_text()).group(1))


GRIDS = {   # name: (cells per axis, tiles compared with the line, line)
    "counts": ((32, 32, 24), "<=", "kScanDirectTiles"),
    "sums": ((32, 32, 25), ">", "kScanDirectTiles"),
    "most sums": ((256, 256, 256), "<=", "kScanSumTiles"),
    "scanned": ((256, 256, 257), ">", "kScanSumTiles"),
}


@pytest.mark.parametrize("name", sorted(GRIDS))
def test_scan_matches_the_oracle(gsph, oracle, cuda_device, name):
    grid, side, line = GRIDS[name]
    _, p, _ = dam_scene(gsph, n_side=2, box=tuple((g - 0.5) * H for g in grid))
    assert tuple(p.grid_size) == grid
    numc = int(np.prod(np.asarray(grid, np.int64)))
    tiles = -(-numc // (constant("kScanThreads") * constant("kScanItems")))
    at = constant(line)
    assert (at - 1 <= tiles <= at) if side == "<=" else (at < tiles <= at + 64)
    rng = np.random.default_rng(3)
    world = np.asarray(grid) * H
    spread = rng.uniform(0.0, 1.0, (20011, 3)) * world               # single particles
    middles = (rng.integers(0, np.asarray(grid), (400, 3)) + 0.5) * H
    small = np.repeat(middles[:300], 20, 0)                          # cells of about 20
    large = np.repeat(middles[300:], 75, 0)                          # and of about 75
    corners = np.array([[0, 0, 0], world - H], np.float64) + H / 2   # first and last cell
    crowd = np.concatenate([small, large, np.repeat(corners, 40, 0)])
    crowd = crowd + rng.uniform(-0.45, 0.45, crowd.shape) * H
    xyz = np.concatenate([spread, crowd]).astype(np.float32)
    xyz = np.clip(xyz, np.float32(1e-5), (world - 1e-3).astype(np.float32))
    pos = np.zeros((len(xyz), 4), np.float32)
    pos[:, :3] = xyz[rng.permutation(len(xyz))]
    with gsph.HybridSystem(params=p, positions=pos) as h:
        h.arrange()
        h.sync()
        key, perm = h.copy_out(gsph.FIELD_KEY), h.copy_out(gsph.FIELD_PERMUTATION)
        start, req = h.copy_out(gsph.FIELD_CELL_START), h.copy_out(gsph.FIELD_BLOCK_REQ)
        compact, split = h.copy_out(gsph.FIELD_COMPACT_INDEX), h.copy_out(gsph.FIELD_SPLIT)
        tasks, info = h.copy_out(gsph.FIELD_TASKS), h.info()
    okey, operm, ostart, bad = oracle.sort(pos, p)
    assert not bad
    assert np.array_equal(start, ostart)
    assert np.array_equal(key, okey) and np.array_equal(perm, operm)
    count = np.diff(ostart)
    assert info.occupied_cells == np.count_nonzero(count)
    assert info.big_cells == np.count_nonzero(count > constant("kSmallCellMax")) > 0
    oreq = oracle.block_req(ostart, p)
    ocompact, middle = oracle.split(ostart, oreq, p)
    otasks = oracle.tasks(okey, ostart, oreq, p, gsph.BLOCK_TASK_DTYPE)
    assert np.array_equal(req, oreq) and np.array_equal(compact, ocompact)
    assert split[0] == middle < len(pos) and split[1] == int(oreq.sum()) > 0
    for f in gsph.BLOCK_TASK_DTYPE.names:
        if f != "pad_":
            assert np.array_equal(tasks[f], otasks[f]), f
