"""The FP64 sweeps with 4 to 32 lanes per particle against one thread each, at
sizes on both sides of every change of the lane count and of a warp's share of
particles: bit for bit (the thread-per-particle sweeps equal the reference)."""
import numpy as np
import pytest

import mphexplicit_b200 as M
from mphexplicit_b200 import scenes
from tests.common import STATE_KEYS, assert_same

pytestmark = pytest.mark.gpu


def droplet(n):
    sc = scenes.droplet_2d(n=int(np.ceil(np.sqrt(n))), seed=n, box=250.0)
    sc.type, sc.xyz, sc.vel = sc.type[:n], sc.xyz[:n], sc.vel[:n]
    sc.header.particle_count = n
    return sc


def dam(fluid, st):
    sc = scenes.dam_break_3d(fluid=fluid, box=tuple(f + 4 for f in fluid), seed=sum(fluid))
    if st:  # every pair term, unequal interaction ratios
        for t in range(4):
            sc.params.surface_tension[t] = 0.05
        sc.params.interaction_ratio[0][2] = 0.8
        sc.params.interaction_ratio[2][0] = 0.7
    return sc


# 2-D lists are short (bounds 6000, 16000, 35000), 3-D whole lists long (2000, 4500, 20000, 60000)
CASES = [("1", lambda: droplet(1)), ("33", lambda: droplet(33))]
CASES += [(f"droplet {n}", lambda n=n: droplet(n)) for n in (6000, 6001, 16000, 16001, 35000, 35001)]
CASES += [(f"dam {f} {st}", lambda f=f, st=st: dam(f, st)) for st in (False, True)
          for f in ((10, 10, 20), (9, 13, 18), (15, 15, 20), (14, 17, 19), (20, 25, 40), (21, 25, 39))]


@pytest.mark.parametrize("name", [n for n, _ in CASES])
def test_lanes_match_thread_sweeps(name):
    sc = dict(CASES)[name]()
    sc.vel[sc.type < 2] += np.random.default_rng(1).normal(size=(sc.n_fluid, 3)) * (0.1, 0.1, 0.1 if sc.dim == 3 else 0)
    got = []
    for layout in ("auto", "thread"):
        s = M.Solver(sc.params, sc.header, sc.type, sc.xyz, sc.vel, dim=sc.dim)
        s.set_sweep_layout(layout)
        s.step(3)
        got.append(s.state())
        s.close()
    for k in STATE_KEYS:
        if k != "virial_pressure":
            assert_same(got[0][k], got[1][k], k)
