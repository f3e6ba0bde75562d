"""Mixed steps launched ahead of the host against one step per call: the same bits,
across rebuilds and in calls of any length."""
import numpy as np
import pytest

import mphexplicit_b200 as M
from mphexplicit_b200 import scenes

pytestmark = pytest.mark.gpu


def droplet():
    sc = scenes.droplet_2d(n=30, seed=5, box=100.0)
    sc.vel[:, 0], sc.vel[:, 1] = 15.0 * sc.xyz[:, 0], -15.0 * sc.xyz[:, 1]
    return sc


def dam():
    sc = scenes.dam_break_3d(fluid=(8, 7, 10), box=(24, 7, 13), seed=4)
    f = sc.type < 2
    sc.vel[f] += np.random.default_rng(2).normal(size=(int(f.sum()), 3)) * 0.5
    return sc


@pytest.mark.parametrize("mode", ["mixed", "mixed_p64", "mixed_walk"])
@pytest.mark.parametrize("make,calls", [(droplet, (2, 37, 1, 90)), (dam, (50, 3)), (dam, (1, 2, 1, 2, 60))])
def test_steps_ahead_match_single_steps(make, calls, mode):
    sc = make()
    a = M.Solver(sc.params, sc.header, sc.type, sc.xyz, sc.vel, dim=sc.dim, mode=mode)
    b = M.Solver(sc.params, sc.header, sc.type, sc.xyz, sc.vel, dim=sc.dim, mode=mode)
    for n in calls:
        a.step(n)
        for _ in range(n):
            b.step(1)
    ia, ib = a.info(), b.info()
    for k in ("step", "time", "rebuild_count"):
        assert ia[k] == ib[k], k
    assert ia["rebuild_count"] > 0
    sa, sb = a.state(), b.state()
    a.close()
    b.close()
    for k in sa:
        if k != "virial_pressure":
            assert np.array_equal(sa[k], sb[k]), k
