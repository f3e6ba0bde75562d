"""The list builds of the FP64 and the mixed form where their split of a cell's
particles over warps changes: one particle, part-filled and full groups of eight, cells
of more than 128 particles (taken in slot order), a table that has to grow, walls
with and without fluid in reach."""
import numpy as np
import pytest

import mphexplicit_b200 as M
from mphexplicit_b200 import scenes
from oracle import pyoracle as po
from tests.common import assert_same

pytestmark = pytest.mark.gpu


def droplet(n, scale=1.0):
    sc = scenes.droplet_2d(n=int(np.ceil(np.sqrt(n))), seed=n, box=100.0)
    sc.type, sc.xyz, sc.vel = sc.type[:n], sc.xyz[:n] * scale, sc.vel[:n]
    sc.header.particle_count = n
    return sc


def dam(fluid, box):
    return scenes.dam_break_3d(fluid=fluid, box=box, seed=sum(fluid))


def crowd():
    """A 3-D dam whose fluid is three times too dense along each axis."""
    sc = dam((12, 12, 12), (36, 12, 16))
    f = sc.type < 2
    sc.xyz[f] = sc.xyz[f] / 3 + 2 * sc.meta["l0"]
    return sc


CASES = {
    "1": lambda: droplet(1), "7": lambda: droplet(7), "33": lambda: droplet(33), "2500": lambda: droplet(2500),
    "2-D, 150 in a cell": lambda: droplet(1600, 0.3),
    "dam": lambda: dam((8, 7, 9), (24, 7, 12)), "crowd": crowd,
    "column": lambda: scenes.two_fluid_column(n=13, seed=3),
}


def brute_counts(sc, xyz, typ):
    """Neighbours within the list radius (+ self; 0: a wall with none of fluid), and
    the particles with a pair so near the radius that FP32 may tell otherwise: the
    hi grid is at most 2^-22 of a cell of about 4 l0, so 1e-5 l0 is ample."""
    p, h = sc.params, sc.header
    l0 = h.particle_spacing
    rm = (max(p.radius_ratio_a, p.radius_ratio_p, p.radius_ratio_v) + 0.1) * l0
    width = np.array([h.domain_max[d] - h.domain_min[d] for d in range(3)])
    n, fluid = len(typ), typ < 2
    cnt, sure = np.zeros(n, int), np.ones(n, bool)
    for i in range(n):
        d = xyz - xyz[i]
        d -= width * np.round(d / width)
        if sc.dim == 2:
            d[:, 2] = 0.0
        r = np.sqrt((d * d).sum(1))
        near = r <= rm
        near[i] = False
        cnt[i] = near.sum() + 1 if fluid[i] or (near & fluid).any() else 0
        sure[i] = not ((np.abs(r - rm) < 1e-5 * l0).any())
    return cnt, sure


@pytest.mark.parametrize("name", list(CASES))
def test_mixed_counts_match_brute_force(name):
    sc = CASES[name]()
    s = M.Solver(sc.params, sc.header, sc.type, sc.xyz, sc.vel, dim=sc.dim, mode="mixed")
    st = s.state()
    s.close()
    want, sure = brute_counts(sc, st["xyz"], st["type"])
    assert sure.mean() > 0.5
    assert np.array_equal(st["neighbor_count"][sure], want[sure])


@pytest.mark.parametrize("name", list(CASES))
def test_fp64_lists_match_the_oracle(name):
    sc = CASES[name]()
    s = M.Solver(sc.params, sc.header, sc.type, sc.xyz, sc.vel, dim=sc.dim)
    o = po.Oracle.from_scene(sc)
    s.step(1)
    o.step(1)
    a, b, la, lb = s.state(), o.state(), s.neighbors(), o.neighbors()
    s.close()
    for k in ("particle_index", "neighbor_count", "density_a", "vol_strain_p", "xyz", "vel"):
        assert_same(a[k], b[k], k)
    assert np.array_equal(la[0], lb[0]) and np.array_equal(la[1], lb[1])
