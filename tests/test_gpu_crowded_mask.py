"""A pair on the edge of interacting, in a particle with more than 64
neighbours. The TRA density pass decides which candidates interact (with its
own rounding of the squared distance) and the force pass follows its masks. In
the smallest scenes, whose force pass lists up to 64 neighbours of a particle,
and in a batch large enough for the general kernels, the decision is the same
and so are the bits. The pair lies 1e-6 apart, where one rounding of the squared
distance reaches the smallest that interacts and the other does not; its
pressure term is as large as any."""
from fractions import Fraction

import numpy as np
import pytest

from gpu_helpers import dam_scene

pytestmark = pytest.mark.gpu

SMALL = np.float32(1e-12)


def rounded(x):
    """The float32 nearest to an exact value (no ties met here)."""
    near = np.float32(float(x))
    around = [np.nextafter(near, np.float32(-1)), near, np.nextafter(near, np.float32(1))]
    return min(around, key=lambda f: abs(Fraction(float(f)) - x))


def edge_pair():
    """Two positions in the plane z = 0.03 that the plain squared distance
    (x^2, then + y^2 fused) takes for interacting and the density pass's form
    (less the smallest distance first, fused) does not."""
    base = np.float32(0.0015)
    unit = 2.0 ** -33                                    # spacing of floats there
    k = int(float(SMALL) ** 0.5 / unit)
    for a in range(k // 2, k):
        b = int((float(SMALL) / unit ** 2 - a * a) ** 0.5)
        for c in (b, b + 1):
            q = np.array([base + np.float32(a * unit), base + np.float32(c * unit)])
            dx, dy = (Fraction(float(v)) - Fraction(float(base)) for v in q)
            plain = rounded(dy * dy + Fraction(float(rounded(dx * dx))))
            less = rounded(dy * dy + Fraction(float(rounded(dx * dx - Fraction(float(SMALL))))))
            if plain >= SMALL and less < 0:
                return base, q
    raise AssertionError("no such pair")


@pytest.mark.parametrize("artificial", [False, True])
def test_an_edge_pair_among_many_neighbours(gsph, cuda_device, artificial):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    _, p, filler = dam_scene(gsph, n_side=int(np.ceil((41 * sms * 32) ** (1 / 3))),
                             box=(1.2, 1.2, 1.2))
    assert len(filler) > 40 * sms * 32
    base, q = edge_pair()
    rng = np.random.default_rng(2)
    cloud = []                                           # 24 neighbours in each z row
    for z0, z1 in ((0.0135, 0.0195), (0.0205, 0.0395), (0.0405, 0.0465)):
        xy = rng.uniform(0.0005, 0.008, (24, 2))
        cloud.append(np.c_[xy, rng.uniform(z0, z1, 24)])
    xyz = np.concatenate([[[base, base, 0.03], [q[0], q[1], 0.03]], *cloud]).astype(np.float32)
    pos = np.zeros((len(xyz), 4), np.float32)
    pos[:, :3] = xyz

    def force(h):
        t = h.get_tuning()
        t.sparse_total = t.sparse_self = 1 << 30         # all TRA
        h.set_tuning(t)
        if artificial:
            h.set_viscosity_model(gsph.VISCOSITY_ARTIFICIAL, 0.02, 20.0)
        ev = h.copy_out(gsph.FIELD_EVAL_VELOCITY)
        ev[:len(pos), :3] = np.random.default_rng(1).normal(0, 1, (len(pos), 3))
        h.copy_in(gsph.FIELD_EVAL_VELOCITY, ev)
        h.arrange()
        h.density()
        count = h.copy_out(gsph.FIELD_NEIGHBOR_COUNT)[:len(pos)]
        h.force()
        return count, h.copy_out(gsph.FIELD_ACCELERATION)[:len(pos)]

    with gsph.HybridSystem(params=p, positions=pos) as h:
        count, alone = force(h)
    with gsph.Batch([(p, pos), (p, filler)]) as b:
        count_b, both = force(b)
    assert np.array_equal(count, count_b) and count.max() > 64
    assert np.array_equal(alone.view(np.uint32), both.view(np.uint32))
