"""The global solve over the merged supernodal tree, at the sizes where its
tiles, chunks and column segments end: one supernode of fewer than 8 columns up
to roots of more than 512 (two segments of v), rows and columns that are no
multiple of 8 or 32. Each step is compared with the FP64 oracle, and every order
of the work, warp-item limit and compiled form must give the same bits."""
import numpy as np
import pytest

import oracle_api as O
from vistio_b200 import api, scenarios

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


def strip(cols, rows):
    px, py, pz, tris = scenarios.quad_grid(cols, rows, cols / max(cols, rows), rows / max(cols, rows))
    pin = np.zeros(len(px), np.uint8)
    pin[: cols + 1] = 1
    return scenarios.Mesh(px, np.ones_like(px), py.copy(), tris, pin)


@pytest.mark.parametrize("cols,rows", [(1, 1), (1, 2), (2, 2), (4, 5), (5, 5), (7, 9), (3, 120), (33, 31), (150, 150)])
@pytest.mark.parametrize("host", [False, True])
def test_step_matches_fp64_in_every_schedule(cols, rows, host):
    if host and cols > 100:
        pytest.skip("the host's numeric factorization of this size is covered by the smaller ones")
    mesh = strip(cols, rows)
    setup = api.SetupDesc(stiffness=1e3, bend_stiffness=1e-4, density_gsm=150.0)
    cfg = api.drape_config(max_iterations=4, host_factorization=host)
    rng = np.random.default_rng(cols * 1000 + rows)
    start = np.stack([mesh.px, mesh.py, mesh.pz], 1)
    start = (start + 1e-3 * rng.uniform(-1, 1, start.shape) * (mesh.pinned == 0)[:, None]).astype(np.float32)
    ref = O.OracleSim(mesh, O.init_params(stiffness=1e3, bend_stiffness=1e-4, density_gsm=150.0),
                      O.default_config(max_iterations=4), precision=1)
    ref.set_state(start.astype(np.float64), np.zeros(start.shape))
    ref.step(DT)
    s = api.ProjectiveDynamicsSolver().init_explicit(mesh, cfg, setup, pinned=mesh.pinned)
    batch = api.Batch([s])
    first = None
    for mode, limit, blocks in [("dataflow", 6144, 2), ("levels", 6144, 4), ("levels", 0, 4), ("dataflow", 0, 5),
                                ("levels", 1024, 5), ("levels", 1 << 30, 2)]:
        batch.set_sweep_mode(mode)
        batch.set_warp_limit(limit)
        batch.set_sweep_blocks(blocks)
        batch.set_state(0, start)
        batch.step(DT)
        got = batch.state(0)[0]
        want = ref.state()[0]
        assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 1e-5
        if first is None:
            first = got
        assert np.array_equal(got, first), (mode, limit, blocks)
