"""The compact index where only some of the model's tiles (1,024 occupied cells
each) hold SMS cells: sparse fluid of several tiles with clumps in the first, a
middle, the last or every tile, or in two cells next to a tile's border, bit for
bit against the oracle's split."""
import numpy as np
import pytest

from gpu_helpers import dam_scene, shuffled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(0,), (1500,), (-1,), (1023, 1024), (1022,), (2048,),
                                   (5, 1100, 2100, -3)])
def test_clumps_in_some_tiles(gsph, oracle, cuda_device, cells):
    _, p, pos = dam_scene(gsph, n_side=33, box=(1.2, 1.0, 0.9))
    with gsph.HybridSystem(params=p, positions=pos) as h:
        h.arrange()
        count = h.copy_out(gsph.FIELD_CELL_COUNT)
        start = h.copy_out(gsph.FIELD_CELL_START)
        spos = h.copy_out(gsph.FIELD_POSITION)
    occupied = np.flatnonzero(count)
    assert len(occupied) > 3 * 1024 and len(occupied) % 32
    # 40 particles more around the first particle of each chosen occupied cell
    rng = np.random.default_rng(7)
    extra = []
    for c in cells:
        at = spos[start[occupied[c]]].copy()
        clump = np.repeat(at[None], 40, axis=0)
        clump[:, :3] += rng.uniform(-1e-4, 1e-4, (40, 3)).astype(np.float32)
        extra.append(clump)
    both = shuffled(np.concatenate([pos] + extra).astype(np.float32))
    with gsph.HybridSystem(params=p, positions=both) as h:
        h.arrange()
        req = h.copy_out(gsph.FIELD_BLOCK_REQ)
        split = h.copy_out(gsph.FIELD_SPLIT)
        compact = h.copy_out(gsph.FIELD_COMPACT_INDEX)
        cs = h.copy_out(gsph.FIELD_CELL_START)
    oreq = oracle.block_req(cs, p)
    ocompact, middle = oracle.split(cs, oreq, p)
    assert np.array_equal(req, oreq)
    assert 0 < middle < len(both) and split[0] == middle
    assert np.array_equal(compact, ocompact)
