"""What a context says and holds once a step has given a non-finite velocity: the state
after as many steps as it counts, and the same call fails as on the path that waits for
every step."""
import numpy as np
import pytest

import mphexplicit_b200 as M
from mphexplicit_b200 import _native as N
from mphexplicit_b200 import scenes

pytestmark = pytest.mark.gpu


def with_nan(sc, k, **kw):
    s = M.Solver(sc.params, sc.header, sc.type, sc.xyz, sc.vel, dim=sc.dim, **kw)
    st = s.state()
    v = st["vel"].copy()
    v[k, 0] = np.nan
    s.set_state(st["xyz"], v)
    return s


def fails(f, *a):
    with pytest.raises(M.MphError) as e:
        f(*a)
    assert e.value.code == N.MPH_ERR_NONFINITE


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_steps_ahead_count_what_ran(mode):
    """Two particles out of each other's reach: the sound one has moved by v dt a step."""
    sc = scenes.droplet_2d(n=2, seed=1)
    l0, dt = sc.header.particle_spacing, sc.params.dt
    sc.type, sc.xyz, sc.vel = sc.type[:2], sc.xyz[:2].copy(), sc.vel[:2].copy()
    sc.header.particle_count = 2
    sc.xyz[1] = sc.xyz[0] + np.array([20.0, 0.0, 0.0]) * l0
    sc.vel[:] = 0.0
    sc.vel[:, 1] = 0.0004 * l0 / dt  # no rebuild within 100 steps
    s = with_nan(sc, 0, mode=mode)
    st = s.state()
    k = int(np.flatnonzero(np.isfinite(st["vel"][:, 0]))[0])
    y, v = st["xyz"][k, 1], st["vel"][k, 1]
    fails(s.step, 60)
    info = s.info()
    assert 0 < info["step"] <= 60 and info["rebuild_count"] == 0
    lo, w = sc.header.domain_min[1], sc.header.domain_max[1] - sc.header.domain_min[1]
    t = 0.0
    for _ in range(info["step"]):
        y = y + v * dt
        y = (y - lo) - w * np.floor((y - lo) / w) + lo
        t += dt
    st = s.state()
    assert st["xyz"][k, 1] == y and st["vel"][k, 1] == v and info["time"] == t
    fails(s.step, 1)
    s.close()


@pytest.mark.parametrize("pinned", [True, False])
def test_read_back_step_fails_where_the_waiting_path_does(pinned):
    """The step that gives the velocity hands it out; the next one fails."""
    import torch
    sc = scenes.droplet_2d(n=12, seed=3)
    a, b = with_nan(sc, 5), with_nan(sc, 5)
    x, v = (torch.zeros((a.n, 3), dtype=torch.float64, pin_memory=pinned).numpy() for _ in range(2))
    xb, vb = np.zeros((b.n, 3)), np.zeros((b.n, 3))
    a.step_read_state(1, x, v)
    b.step(1)
    b.get_xv(xb, vb)
    assert np.isnan(vb).any()
    assert np.array_equal(x, xb, equal_nan=True) and np.array_equal(v, vb, equal_nan=True)
    fails(a.step_read_state, 1, x, v)
    fails(b.step, 1)
    a.get_xv(x, v)
    b.get_xv(xb, vb)
    assert np.array_equal(x, xb, equal_nan=True) and np.array_equal(v, vb, equal_nan=True)
    ia, ib = a.info(), b.info()
    assert ia["step"] == ib["step"] == 1 and ia["time"] == ib["time"]
    a.close()
    b.close()
