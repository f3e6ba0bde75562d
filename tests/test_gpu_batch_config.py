"""A batch whose set_tiles was refused steps on as it was: the same bits as one that was
never asked, in the table form and with tiles, in graph launches and single steps."""
import numpy as np
import pytest

import mphexplicit_b200 as M
from mphexplicit_b200 import scenes

pytestmark = pytest.mark.gpu


def block(seed):
    """Fluid in the corner of a periodic box of 40 cells a side."""
    sc = scenes.dam_break_3d(fluid=(9, 8, 10), box=(20, 12, 14), seed=seed)
    f = sc.type < 2
    sc.type, sc.xyz, sc.vel = sc.type[f], sc.xyz[f], sc.vel[f]
    sc.header.particle_count = len(sc.type)
    for d in range(3):
        sc.header.domain_max[d] = sc.header.domain_min[d] + 40 * 3.7 * sc.header.particle_spacing
    sc.vel += np.random.default_rng(seed).normal(size=sc.vel.shape) * 0.3
    return sc


@pytest.mark.parametrize("start", [None, (1, 1, 1, 64), (1, 1, 1, 256), (2, 2, 4, 128)])
@pytest.mark.parametrize("threads", [64, 256])
def test_refused_tiles_change_nothing(start, threads):
    scs = [block(s) for s in (1, 2, 3)]
    a, b = M.Batch(scs, tiles=start), M.Batch(scs, tiles=start)
    for steps in (3, 40):  # direct launches; graph launches and a remainder
        with pytest.raises(M.MphError):
            b.set_tiles(32, 32, 32, threads)  # the halo's tables alone exceed an SM's shared memory
        a.step(steps)
        b.step(steps)
        assert a.info() == b.info()
        for x, y in zip(a.state(), b.state()):
            assert np.array_equal(x, y)
    a.close()
    b.close()
