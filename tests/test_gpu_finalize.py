"""Faces in cell order and the cell -> face CSR, from the faces themselves: at the sizes
where a scan takes one block, two launches or three, for cells with more incoming faces
than a group of lanes ranks, and for batches and masked builds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check_csr(v):
    n, left, right = v.n_cells, np.asarray(v.face_left), np.asarray(v.face_right)
    assert np.all(np.diff(left) >= 0)
    linked = np.flatnonzero((right >= 0) & (np.asarray(v.face_shift_code) == 13))
    cell = np.concatenate([left, right[linked]])
    face = np.concatenate([np.arange(len(left)), linked])
    count = np.bincount(cell, minlength=n)
    assert np.array_equal(v.cell_face_count, count)
    assert np.array_equal(v.cell_face_offset, np.cumsum(count) - count)
    assert np.array_equal(v.cell_face_connections, face[np.lexsort((face, cell))])


@pytest.mark.parametrize("n", [1, 2, 4095, 16384, 16385, 70_000, 8_400_000, 9_000_000])
@pytest.mark.parametrize("periodic", [False, True])
def test_csr_1d(gpu_ctx, n, periodic):
    """1-D: the largest n, and the faces are known (each cell's neighbours)."""
    rng = np.random.default_rng(n)
    place = rng.permutation(n)
    g = np.zeros((n, 3))
    g[:, 0] = (place + 0.5 + 0.2 * rng.random(n)) / n
    v = gpu_ctx.build_arrays(g, None, [0, 0, 0], [1, 1, 1], 1, periodic)
    assert np.all(np.asarray(v.cell_face_count) <= 2)
    check_csr(v)


@pytest.mark.parametrize("dim,n", [(2, 3000), (2, 40_000), (3, 1000), (3, 30_000)])
def test_csr(gpu_ctx, dim, n):
    rng = np.random.default_rng(n)
    g = rng.random((n, 3))
    g[:, dim:] = 0.0
    mask = rng.random(n) < 0.6
    for m, periodic in ((None, True), (None, False), (mask, True)):
        check_csr(gpu_ctx.build_arrays(g, m, [0, 0, 0], [1, 1, 1], dim, periodic))


@pytest.mark.parametrize("star", [8, 30, 31, 32, 33, 34, 60, 90])
def test_many_incoming_faces(gpu_ctx, star):
    """The last generator is the right cell of all its neighbours on a circle."""
    rng = np.random.default_rng(star)
    a = 2.0 * np.pi * (np.arange(star) + 0.1 * rng.random(star)) / star
    ring = np.stack([0.5 + 0.2 * np.cos(a), 0.5 + 0.2 * np.sin(a), 0.0 * a], axis=1)
    far = rng.random((400, 3)) * [1, 0.15, 0]
    g = np.concatenate([rng.permutation(ring), far, [[0.5, 0.5, 0.0]]])
    v = gpu_ctx.build_arrays(g, None, [0, 0, 0], [1, 1, 1], 2, False)
    assert v.cell_face_count[-1] == star
    check_csr(v)


def test_csr_batch(gpu_ctx):
    rng = np.random.default_rng(3)
    jobs = []
    for n in (1, 700, 5000, 20_000):
        jobs.append(dict(generators=rng.random((n, 3)), anchor=[0, 0, 0], width=[1, 1, 1], dimensionality=3,
                         periodic=n > 1))
    for j, v in zip(jobs, gpu_ctx.build_batch(jobs)):
        check_csr(v)
        alone = gpu_ctx.build_arrays(j["generators"], None, j["anchor"], j["width"], 3, j["periodic"])
        assert np.array_equal(v.cell_face_connections, alone.cell_face_connections)
