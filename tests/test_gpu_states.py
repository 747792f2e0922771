"""A garment's state after several steps against the state that earlier builds of
this library gave for it (tests/golden/strip_states.npz: positions and velocities
before and after). v = (x - x_prev) / dt multiplies a last bit of a position by
1 / dt, and the stiff elements feed it back: a solve whose sums round in another
way, though no less exactly, moves these velocities by 3.3e-5 of their norm."""
import os

import numpy as np

import pytest

from vistio_b200 import api, scenarios

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "strip_states.npz")
BOUND = 2e-5  # of the 2-norm: what a float32 result may move between builds


@pytest.mark.parametrize("batched", [False, True])
def test_strip_states_are_those_of_earlier_builds(batched):
    cols, rows = 104, 13
    px, py, pz, tris = scenarios.quad_grid(cols, rows, 1.0, rows / cols)
    pinned = np.zeros(len(px), np.uint8)
    pinned[: cols + 1] = 1
    mesh = scenarios.Mesh(px, np.ones_like(px), py.copy(), tris, pinned)
    setup = api.SetupDesc(model=2, bending=3, stiffness=1248.2001249293255, bend_stiffness=3.978409131307211e-05,
                          density_gsm=97.06005335638419, warp_stiffness=0.9, weft_stiffness=0.6, bend_warp=0.9,
                          bend_weft=0.4)
    s = api.ProjectiveDynamicsSolver().init_explicit(mesh, api.drape_config(max_iterations=10), setup, pinned=pinned)
    run = np.load(GOLDEN)
    if batched:
        b = api.Batch([s])
        b.set_state(0, run["pos"], run["vel"])
        b.step(1.0 / 60.0, 4)
        pos, vel = b.state(0)
    else:
        s.set_state(run["pos"], run["vel"])
        for _ in range(4):
            s.step(1.0 / 60.0)
        pos, vel = s.state()
    for got, want in ((pos, run["pos_after"]), (vel, run["vel_after"])):
        assert np.linalg.norm(got.astype(np.float64) - want) <= BOUND * np.linalg.norm(want.astype(np.float64))
