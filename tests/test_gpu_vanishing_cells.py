"""Cuts that remove all of a cell's vertices: a generator outside a closed box, whose bisectors
leave nothing of the box on its side.  The reference's loop makes a ring of two nodes of
such a region and goes on with two vertices (or fails on them); results, errors and their
cells have to be the oracle's, bit for bit."""
import numpy as np
import pytest

from meshless_voro_b200._native import MvError

pytestmark = pytest.mark.gpu
BOX = ([0, 0, 0], [1, 1, 1])


def _check(gpu_ctx, oracle, g, mask, dim, precision):
    orc = oracle.build(g, *BOX, dim=dim, periodic=False, mask=mask)
    kw = dict(precision=precision, pipeline="staged")
    if orc.status == 0:
        gpu = gpu_ctx.build_arrays(g, mask, *BOX, dim, False, **kw)
        for a, b in [(gpu.cell_volume, orc.volume), (gpu.cell_centroid, orc.centroid),
                     (gpu.cell_safety_radius, orc.safety_radius), (gpu.face_left, orc.face_left),
                     (gpu.face_right, orc.face_right), (gpu.face_area, orc.face_area),
                     (gpu.face_centroid, orc.face_centroid), (gpu.face_normal, orc.face_normal),
                     (gpu.cell_face_offset, orc.face_offset), (gpu.cell_face_count, orc.face_count),
                     (gpu.cell_face_connections, orc.cell_face_connections)]:
            assert np.array_equal(a, b)
        return
    with pytest.raises(MvError) as e:
        gpu_ctx.build_arrays(g, mask, *BOX, dim, False, **kw)
    assert (e.value.status, e.value.error_cell) == (orc.status, orc.error_cell)


@pytest.mark.parametrize("precision", ["filtered", "fp64"])
@pytest.mark.parametrize("dim,seed", [(d, s) for d in (1, 2, 3) for s in range(8)])
def test_generators_outside_a_closed_box(gpu_ctx, oracle, dim, seed, precision):
    rng = np.random.default_rng(seed)
    g = rng.random(((0, 12, 60, 300)[dim], 3))
    g[:, dim:] = 0.0
    for i in range(3):
        d = rng.uniform(0.05, 0.3)
        g[i, rng.integers(0, dim)] = rng.choice([-d, 1.0 + d])
    out = np.arange(len(g)) < 3
    for i in range(3):  # one at a time, so that an error is that cell's
        _check(gpu_ctx, oracle, g, np.arange(len(g)) == i, dim, precision)
    _check(gpu_ctx, oracle, g, ~out, dim, precision)


@pytest.mark.parametrize("precision", ["filtered", "fp64"])
def test_first_cut_takes_the_whole_box(gpu_ctx, oracle, precision):
    _check(gpu_ctx, oracle, np.array([[0.5, 0.5, 0.5], [-0.9, 0.5, 0.5]]), None, 3, precision)
    for n in (300, 9000):  # the wide tier and the first
        g = np.random.default_rng(1).random((n, 3))
        g[7] = [-2.0 * n ** (-1.0 / 3.0), 0.5, 0.5]
        _check(gpu_ctx, oracle, g, None, 3, precision)
