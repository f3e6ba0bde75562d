"""The batched form's neighbour table against its tile sweeps.

Both visit a particle's pairs in the same order with the same expressions.  In
2-D the table form rounds every displacement as a tile of the default shape
does, so the two agree to the bit.  In 3-D the long pairs' displacements are
rounded once from FP64: a pair's force then differs by at most one FP32
rounding of its displacement (2^-24), and so does the velocity, which is a sum
of such terms: 1e-7 relative.
"""
import numpy as np
import pytest

import mphexplicit_b200 as M
from mphexplicit_b200 import scenes
from tests.common import rel_l2
from tests.test_gpu_batch import small_dams, small_droplets

pytestmark = pytest.mark.gpu

TILES = {2: (8, 8, 1, 256), 3: (2, 2, 4, 256)}  # the default tiles


def squeezed(dim):
    """Lists far longer than their tables (sized for the lattice spacing):
    every particle is walked from the cells."""
    if dim == 2:
        sc = scenes.droplet_2d(n=30, seed=4)
    else:
        sc = scenes.dam_break_3d(fluid=(8, 8, 8), box=(20, 12, 14), seed=4)
    f = sc.type < 2
    c = sc.xyz[f].mean(axis=0)
    sc.xyz[f] = c + 0.55 * (sc.xyz[f] - c)
    return [sc]


def across_faces(dim):
    """Fluid around every corner of the periodic domain, drifting through its faces."""
    if dim == 2:
        sc = scenes.droplet_2d(n=24, seed=6, box=40.0)
    else:
        sc = scenes.dam_break_3d(fluid=(10, 10, 10), box=(14, 14, 14), seed=6)
        keep = sc.type < 2
        sc.type, sc.xyz, sc.vel = sc.type[keep], sc.xyz[keep], sc.vel[keep]
        sc.header.particle_count = len(sc.type)
    lo = np.array([sc.header.domain_min[d] for d in range(3)])
    hi = np.array([sc.header.domain_max[d] for d in range(3)])
    sc.xyz[:, :dim] = lo[:dim] + np.mod(sc.xyz[:, :dim] - sc.xyz[:, :dim].mean(axis=0), (hi - lo)[:dim])
    sc.vel[:, :dim] = 3.0
    return [sc]


def one_particle(dim):
    scs = small_droplets(count=2, seed=31) if dim == 2 else small_dams(count=2, seed=31)
    sc = scs[0]
    k = int(np.flatnonzero(sc.type < 2)[0])
    sc.type, sc.xyz, sc.vel = sc.type[k:k + 1], sc.xyz[k:k + 1], sc.vel[k:k + 1]
    sc.header.particle_count = 1
    return scs


CASES = {"plain": lambda d: small_droplets(5, 23) if d == 2 else small_dams(4, 23), "squeezed": squeezed,
         "faces": across_faces, "one": one_particle}
STEPS = {"plain": 70, "squeezed": 2, "faces": 40, "one": 20}


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("name", list(CASES))
def test_table_matches_tile_sweeps(name, dim):
    scs, steps = CASES[name](dim), STEPS[name]
    got = []
    for tiles in (None, TILES[dim]):
        b = M.Batch(scs, tiles=tiles)
        b.step(steps)
        got.append(b.state())
        assert (b.info()["tile"] == (1, 1, 1)) == (tiles is None)
        b.close()
    (x, v), (xt, vt) = got
    assert np.any(vt != 0.0)
    if dim == 2:
        assert np.array_equal(x, xt) and np.array_equal(v, vt)
    else:
        assert rel_l2(v, vt) < 1e-7 and rel_l2(x, xt) < 1e-7


@pytest.mark.parametrize("dim", [2, 3])
def test_switching_between_table_and_tiles(dim):
    """A batch that leaves the table form and comes back steps as one that
    stayed (2-D: to the bit, across sorts in the tile form too)."""
    scs = CASES["plain"](dim)
    a = M.Batch(scs)
    a.step(90)
    b = M.Batch(scs)
    b.step(30)
    b.set_tiles(*TILES[dim])
    b.step(30)
    b.set_tiles(1, 1, 1, 128)
    b.step(30)
    (xa, va), (xb, vb) = a.state(), b.state()
    a.close()
    b.close()
    if dim == 2:
        assert np.array_equal(xa, xb) and np.array_equal(va, vb)
    else:
        assert rel_l2(vb, va) < 1e-6 and rel_l2(xb, xa) < 1e-7  # 30 of 90 steps in the other form
