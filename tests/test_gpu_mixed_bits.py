"""The mixed form's sweeps by one and by several lanes per particle: the same sums in
the same order, so the same bits, and those that a thread per particle has always given:
tests/golden/mixed_bits.json keeps digests of the state after some steps of small scenes."""
import hashlib
import json
import os

import numpy as np
import pytest

import mphexplicit_b200 as M
from mphexplicit_b200 import scenes

pytestmark = pytest.mark.gpu

KEYS = ("particle_index", "xyz", "vel", "force", "density_a", "vol_strain_p")
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "mixed_bits.json")


def droplet(n):
    sc = scenes.droplet_2d(n=n, seed=n, box=100.0)
    sc.vel[:, 0], sc.vel[:, 1] = 15.0 * sc.xyz[:, 0], -15.0 * sc.xyz[:, 1]
    return sc


def dam(fluid, st=False):
    sc = scenes.dam_break_3d(fluid=fluid, box=(2 * fluid[0], fluid[1], fluid[2] + 4), seed=sum(fluid))
    if st:  # every pair term, unequal interaction ratios
        for t in range(4):
            sc.params.surface_tension[t] = 0.05
        sc.params.interaction_ratio[0][2] = 0.8
        sc.params.interaction_ratio[2][0] = 0.7
    return sc


def column(n):
    sc = scenes.two_fluid_column(n=n, seed=n)
    sc.params.shear_viscosity[1] *= 1.5
    return sc


# by size (lanes of the density / force sweep)
SCENES = {"droplet 1": lambda: droplet(1), "droplet 7": lambda: droplet(7), "droplet 92": lambda: droplet(92),  # 8 / 8
          "droplet 150": lambda: droplet(150),                                                                  # 4 / 4
          "dam": lambda: dam((9, 10, 11)), "dam middle": lambda: dam((16, 16, 20)),                             # 8 / 8, 4 / 8
          "dam large": lambda: dam((34, 33, 41)),                                                               # 1 / 4
          "dam st": lambda: dam((11, 9, 12), True), "column": lambda: column(13),                               # 8 / 8
          "column middle": lambda: column(30)}                                                                  # 4 / 4
STEPS = 12


def run(name, mode, layout=None):
    sc = SCENES[name]()
    f = sc.type < 2
    sc.vel[f] += np.random.default_rng(3).normal(size=(int(f.sum()), 3)) * (0.5, 0.5, 0.5 if sc.dim == 3 else 0)
    s = M.Solver(sc.params, sc.header, sc.type, sc.xyz, sc.vel, dim=sc.dim, mode=mode)
    if layout is not None:
        s.set_sweep_layout(layout)
    s.step(STEPS)
    st, rebuilds = s.state(), s.info()["rebuild_count"]
    s.close()
    return st, rebuilds


def digest(st):
    return hashlib.sha256(b"".join(np.ascontiguousarray(st[k]).tobytes() for k in KEYS)).hexdigest()


MODES = ["mixed", "mixed_p64", "mixed_walk"]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("name", list(SCENES))
def test_kept_digests(name, mode):
    st, _ = run(name, mode)
    assert digest(st) == json.load(open(GOLDEN))["%s, %s" % (name, mode)]


@pytest.mark.parametrize("mode", MODES[:2])
@pytest.mark.parametrize("name", list(SCENES))
def test_lane_counts_give_the_same_bits(name, mode):
    a, ra = run(name, mode, "thread")
    for layout in ("auto", "warp"):
        b, rb = run(name, mode, layout)
        assert ra == rb
        for k in KEYS:
            assert np.array_equal(a[k], b[k], equal_nan=True), (layout, k)
    assert ra > 0 or name in ("droplet 1", "droplet 7")
