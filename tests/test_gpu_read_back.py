"""mph_step_read_state against step + get_state: the same bits, and across a rebuild too the
positions are packed and sent once.  With pinned memory the force sweep stores the
velocities to the host itself, a thread or several lanes per particle."""
import numpy as np
import pytest

import mphexplicit_b200 as M
from mphexplicit_b200 import scenes

pytestmark = pytest.mark.gpu

# fluid block, box, particles: over 60,000 fluid ones, a thread each; 8,000 among walls, 8 lanes each; few
SCENES = {"fluid": ((40, 40, 40), (60, 40, 50), 114016), "walls": ((20, 20, 20), (120, 100, 20), 115256),
          "small": ((9, 7, 8), (20, 9, 11), None)}


@pytest.mark.parametrize("pinned", [(True, True), (True, False), (False, True), (False, False)])
@pytest.mark.parametrize("name", list(SCENES))
def test_read_back_is_step_then_get_state(name, pinned):
    import torch
    fluid, box, n = SCENES[name]
    sc = scenes.dam_break_3d(fluid=fluid, box=box, seed=2)
    assert n is None or sc.n == n
    f = sc.type < 2
    sc.vel[f, 2] = 0.02 * sc.header.particle_spacing / sc.params.dt  # 0.05 spacings, a rebuild, in three steps
    a, b = (M.Solver(sc.params, sc.header, sc.type, sc.xyz, sc.vel, dim=3) for _ in range(2))
    x, v = (torch.zeros((sc.n, 3), dtype=torch.float64, pin_memory=p).numpy() for p in pinned)
    xb, vb = np.zeros((sc.n, 3)), np.zeros((sc.n, 3))
    rebuilds = 0
    for _ in range(5):
        la, lb = a.launch_count(), b.launch_count()
        a.step_read_state(1, x, v)
        b.step(1)
        la, lb = a.launch_count() - la, b.launch_count() - lb
        b.get_xv(xb, vb)
        assert np.array_equal(x, xb) and np.array_equal(v, vb)
        r = b.info()["rebuild_count"]
        # beside the step's own: two sweeps that found the step stopped, a pack of the
        # positions and one of velocities that the sweep could not store
        assert la - lb == 1 + (not pinned[1]) + 2 * (r - rebuilds)
        rebuilds = r
    assert rebuilds > 0
    assert a.info()["rebuild_count"] == rebuilds
    a.close()
    b.close()
