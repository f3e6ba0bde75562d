"""The mixed sweeps with 8, 4 and 1 lanes per particle, at sizes on both sides of every
change of the lane count: one step's change of velocity against the FP64 form's."""
import numpy as np
import pytest

import mphexplicit_b200 as M
from mphexplicit_b200 import scenes
from tests.common import by_original_id

pytestmark = pytest.mark.gpu

# A pair term has about ten FP32 roundings (6e-7 relative) and the terms of a force
# cancel to about a hundredth of their size: 6e-5; a list entry left out or taken twice
# changes a force by some 5e-3 or more.
TOL = 1e-3


def droplet(n):
    sc = scenes.droplet_2d(n=int(np.ceil(np.sqrt(n))), seed=n, box=450.0)
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


CASES = [(f"droplet {n}", lambda n=n: droplet(n)) for n in (1, 33, 15000, 15001, 45000, 45001)]
CASES += [(f"dam {f} {st}", lambda f=f, st=st: dam(f, st)) for st in (False, True)
          for f in ((9, 10, 11), (26, 26, 26), (27, 26, 26), (40, 41, 40), (46, 47, 46), (46, 46, 48), (53, 53, 53),
                    (53, 53, 54), (58, 58, 59), (58, 58, 60))]


@pytest.mark.parametrize("mode", ["mixed", "mixed_p64"])
@pytest.mark.parametrize("name", [n for n, _ in CASES])
def test_step_matches_fp64(name, mode):
    sc = dict(CASES)[name]()
    f = sc.type < 2
    sc.vel[f] += np.random.default_rng(1).normal(size=(int(f.sum()), 3)) * (0.1, 0.1, 0.1 if sc.dim == 3 else 0)
    dv = []
    for md in ("fp64", mode):
        s = M.Solver(sc.params, sc.header, sc.type, sc.xyz, sc.vel, dim=sc.dim, mode=md)
        s.step(1)
        st = s.state()
        s.close()
        dv.append(by_original_id(st, "vel")[f] - sc.vel[f])
    scale = np.abs(dv[0]).max()
    assert np.abs(dv[1] - dv[0]).max() <= TOL * max(scale, 1e-12)
