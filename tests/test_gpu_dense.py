"""Shells that reach dense grid cells: clumps of the sizes where a warp's search of a cell
changes its step, inside a cell, across its faces and with generators on the faces of the
cell's octree; rows of cells that alternate between dense and sparse; batches that mix
tessellations with and without dense cells.  Every value has to be the oracle's."""
import numpy as np
import pytest

from voronoi_checks import compare

pytestmark = pytest.mark.gpu


def _clumps(rng, dim, n_background, sizes, spread, snap):
    """A uniform background and clumps; snap: half of a clump's coordinates are multiples of
    2^-12 (faces of the octree cells of a unit box with a power of two of grid cells)."""
    g = [rng.random((n_background, 3))]
    for k, m in enumerate(sizes):
        c = rng.random(3) if k % 2 else np.round(8 * rng.random(3)) / 8.0
        p = c + spread * rng.normal(size=(m, 3))
        if snap:
            on = rng.random((m, 3)) < 0.5
            on[:, 0] = False  # one free coordinate: no two generators alike
            p[on] = np.round(p[on] * 4096.0) / 4096.0
        g.append(p - np.floor(p))
    g = np.concatenate(g)
    g[:, dim:] = 0.0
    return g[rng.permutation(len(g))]


@pytest.mark.parametrize("snap", [False, True])
@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("dim,sizes,spread", [
    (1, (33, 70, 400), 1e-4),
    (2, (33, 64, 65, 96, 97, 900), 2e-3),
    (3, (33, 63, 64, 65, 128, 1025, 2500), 1e-2),
    (3, (60,) * 25, 2e-2),       # many small dense cells between sparse ones
    (3, (40, 3000), 1e-5),       # a clump deep in its cell's octree
])
def test_clumps(gpu_ctx, oracle, dim, sizes, spread, periodic, snap):
    rng = np.random.default_rng(100 * dim + len(sizes))
    g = _clumps(rng, dim, 1500, sizes, spread, snap and spread > 1e-3)
    box = ([0, 0, 0], [1, 1, 1])
    orc = oracle.build(g, *box, dim=dim, periodic=periodic)
    for pipeline in ("staged", "fused"):
        assert compare(gpu_ctx.build_arrays(g, None, *box, dim, periodic, pipeline=pipeline), orc)


def test_batch_of_both(gpu_ctx, oracle):
    rng = np.random.default_rng(8)
    jobs = []
    for k in range(6):
        g = _clumps(rng, 3, 700, (50, 600), 5e-3, False) if k % 2 else rng.random((900, 3))
        jobs.append(dict(generators=g, anchor=[0, 0, 0], width=[1, 1, 1], dimensionality=3, periodic=k < 4))
    for j, v in zip(jobs, gpu_ctx.build_batch(jobs)):
        assert compare(v, oracle.build(j["generators"], j["anchor"], j["width"], dim=3, periodic=j["periodic"]))
