"""Where a size decides which kernels run: both sides of each line against the
FP64 or FP32 oracle, or bit for bit against the garment alone."""
import numpy as np
import pytest

import oracle_api as O
from vistio_b200 import api

from test_gpu_solve import strip

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


def soup(n, size, seed):
    """n triangles of their own vertices, their centres in the unit cube."""
    rng = np.random.default_rng(seed)
    c = rng.uniform(0, 1, (n, 1, 3))
    pos = (c + size * rng.uniform(-0.5, 0.5, (n, 3, 3))).reshape(-1, 3).astype(np.float32)
    return pos, np.arange(3 * n, dtype=np.uint32).reshape(n, 3)


# one leaf and no tree; trees of fewer levels than the traversal starts from; the
# last triangle count of the shared traversal (148 * 512 = 75,776) and the first of the other
@pytest.mark.parametrize("n,size", [(1, 0.5), (2, 6.0), (3, 6.0), (31, 0.5), (33, 0.5), (600, 0.2),
                                    (75776, 0.012), (75777, 0.012)])
def test_broadphase_sizes(n, size):
    pos, tris = soup(n, size, n)
    ref = O.tri_pairs(pos, tris, 1e-3, mode=0)
    got = api.broadphase_pairs(pos, tris, 1e-3)
    assert np.array_equal(got, ref)
    if n <= 65536:  # what that entry point takes
        assert np.array_equal(api.broadphase_pairs_noalloc(pos, tris, 1e-3), ref)


@pytest.mark.parametrize("n", [64, 65, 66, 300])
def test_broadphase_all_overlap(n):
    """Every triangle meets every other: rows of up to n - 1 partners (sorted in
    another way past 64), and for 300 more pairs than the first call has room for."""
    pos, tris = soup(n, 3.0, n)
    pos = (0.01 * pos + np.tile([[0, 0, 0], [1, 0, 0], [0, 1, 0.5]], (n, 1))).astype(np.float32)
    ref = O.tri_pairs(pos, tris, 1e-3, mode=0)
    assert len(ref) == n * (n - 1) // 2
    assert np.array_equal(api.broadphase_pairs(pos, tris, 1e-3), ref)
    assert np.array_equal(api.broadphase_pairs_noalloc(pos, tris, 1e-3), ref)


@pytest.mark.parametrize("count", [2, 60])
def test_batched_steps_bitwise_equal_the_garment_alone(count):
    """A garment alone runs its local steps in one launch and a tile per warp in
    the sweeps; two garments still do; 60 (more than 4 * 148 * 32 tasks in the
    leaves' phase) have a launch per local step and whole supernodes of up to two
    chunks of columns per warp."""
    mesh = strip(64, 61)
    setup = api.SetupDesc(stiffness=1e3, bend_stiffness=1e-4, density_gsm=150.0)
    cfg = api.drape_config(max_iterations=3)
    rng = np.random.default_rng(count)
    start = np.stack([mesh.px, mesh.py, mesh.pz], 1)
    start = (start + 1e-3 * rng.uniform(-1, 1, start.shape) * (mesh.pinned == 0)[:, None]).astype(np.float32)

    def run(n, mode, blocks):
        solvers = [api.ProjectiveDynamicsSolver().init_explicit(mesh, cfg, setup, pinned=mesh.pinned) for _ in range(n)]
        b = api.Batch(solvers)
        b.set_sweep_mode(mode)
        b.set_sweep_blocks(blocks)
        for k in range(n):
            b.set_state(k, start)
        b.step(DT)
        return [b.state(k)[0] for k in (0, n // 2, n - 1)]

    alone = run(1, "levels", 2)[0]
    for mode, blocks in [("levels", 4), ("levels", 5), ("dataflow", 4), ("grouped", 4)]:
        if mode == "grouped" and count < 32:
            continue  # two garments are no group
        for got in run(count, mode, blocks):
            assert np.array_equal(got, alone), (mode, blocks)


def test_local_shapes_that_are_set_are_run():
    """A small batch runs both local steps in one launch until the caller sets
    their shapes: then each is a launch of its own, one more per iteration."""
    mesh = strip(12, 12)
    cfg = api.drape_config(max_iterations=6)
    solvers = [api.ProjectiveDynamicsSolver().init_explicit(mesh, cfg, api.SetupDesc(), pinned=mesh.pinned) for _ in range(2)]
    batch = api.Batch(solvers)
    batch.step(DT)
    launches, want = batch.launches_per_step(), batch.state(0)[0]
    for shape in ((1, 1), (2, 2), (1, 2), (2, 1)):
        batch.set_local_shape(*shape)
        for k in range(2):
            batch.set_state(k, np.stack([mesh.px, mesh.py, mesh.pz], 1))
        batch.step(DT)
        assert batch.launches_per_step() == launches + 6, shape
        assert np.array_equal(batch.state(0)[0], want), shape
