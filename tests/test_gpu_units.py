"""Sweeps by units (a small factor) against the other kernels, at the sizes where a
unit's parts change: supernodes of more than 32 columns, of column sums in parts, of
diagonal products in parts, too large for shared memory; one unit, many, and a batch
whose factor is too large for units."""
import numpy as np
import pytest

from vistio_b200 import api

from test_gpu_solve import strip

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


def start_of(mesh, seed):
    pos = np.stack([mesh.px, mesh.py, mesh.pz], 1)
    rng = np.random.default_rng(seed)
    return (pos + 1e-3 * rng.uniform(-1, 1, pos.shape) * (mesh.pinned == 0)[:, None]).astype(np.float32)


# 64x61 and 97x13: sums in parts; 97x97: a split diagonal product; 128x40, 190x60: chains
# of wide supernodes; 200x200: supernodes of more than 224 KB
@pytest.mark.parametrize("cols,rows,refine", [(12, 9, 0), (64, 61, 1), (97, 13, 0), (97, 97, 2), (128, 40, 0), (190, 60, 0),
                                              (200, 200, 0)])
def test_units_bitwise_equal_levels(cols, rows, refine):
    mesh = strip(cols, rows)
    cfg = api.drape_config(max_iterations=3, refinement_sweeps=refine)
    setup = api.SetupDesc(stiffness=1e3, bend_stiffness=1e-4, density_gsm=150.0)
    batch = api.Batch([api.ProjectiveDynamicsSolver().init_explicit(mesh, cfg, setup, pinned=mesh.pinned)])
    start, got = start_of(mesh, cols), {}
    for mode in ("levels", "dataflow"):
        batch.set_sweep_mode(mode)
        batch.set_state(0, start)
        batch.step(DT, 2)
        got[mode] = batch.state(0)
    for a, b in zip(got["levels"], got["dataflow"]):
        assert np.array_equal(a, b)


def test_batch_too_large_for_units_equals_the_garment_alone():
    """160 sheets, each of more than 1 MB of factor, are past 128 MiB: k_sweep; alone,
    units."""
    mesh = strip(64, 64)
    cfg = api.drape_config(max_iterations=3)
    setup = api.SetupDesc(stiffness=1e3, bend_stiffness=1e-4, density_gsm=150.0)
    start = start_of(mesh, 5)

    def run(n):
        solvers = [api.ProjectiveDynamicsSolver().init_explicit(mesh, cfg, setup, pinned=mesh.pinned) for _ in range(n)]
        batch = api.Batch(solvers)
        batch.set_sweep_mode("dataflow")
        for k in range(n):
            batch.set_state(k, start)
        batch.step(DT)
        return batch, [batch.state(k)[0] for k in (0, n // 2, n - 1)]

    alone, (want, _, _) = run(1)
    many, got = run(160)
    assert alone.info()["factor_bytes"] < 128 << 20 < many.info()["factor_bytes"]
    assert many.launches_per_step() < alone.launches_per_step() + 3  # one launch for both sweeps
    for g in got:
        assert np.array_equal(g, want)


@pytest.mark.parametrize("n", [1, 31, 257, 700, 1600])
def test_dense_matrix(n):
    """Supernodes of 256 columns and up to 1,344 rows: with 700 they pass through
    shared memory, with 1,600 a unit of one does not fit and k_sweep takes the matrix."""
    rng = np.random.default_rng(n)
    a = rng.uniform(-1, 1, (n, n)).astype(np.float32)
    a = ((a + a.T) / 2).astype(np.float32)
    a[np.arange(n), np.arange(n)] = np.float32(n)  # diagonally dominant
    ptr = (np.arange(n + 1) * n).astype(np.uint32)
    col = np.tile(np.arange(n), n).astype(np.uint32)
    s = api.SparseSolver()
    s.factorize(ptr, col, a.ravel(), n)
    b = rng.normal(size=n).astype(np.float32)
    want = np.linalg.solve(a.astype(np.float64), b.astype(np.float64))
    assert np.linalg.norm(s.solve(b) - want) <= 1e-6 * np.linalg.norm(want)


@pytest.mark.parametrize("blocks,size", [(1, 1), (300, 1), (257, 7), (40, 33)])
def test_matrix_of_independent_blocks(blocks, size):
    """Whole trees that share a unit: tridiagonal blocks."""
    n = blocks * size
    i = np.arange(n)
    left, right = i % size > 0, i % size < size - 1
    rows = np.concatenate([i, i[left], i[right]])
    cols = np.concatenate([i, i[left] - 1, i[right] + 1])
    vals = np.concatenate([3.0 + (i % 5), np.full(left.sum() + right.sum(), -1.0)]).astype(np.float32)
    order = np.lexsort((cols, rows))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.uint32)
    s = api.SparseSolver()
    s.factorize(ptr, cols[order].astype(np.uint32), vals[order], n)
    a = np.zeros((n, n))
    a[rows, cols] = vals
    b = np.random.default_rng(n).normal(size=n).astype(np.float32)
    want = np.linalg.solve(a, b.astype(np.float64))
    assert np.linalg.norm(s.solve(b) - want) <= 1e-6 * np.linalg.norm(want)
