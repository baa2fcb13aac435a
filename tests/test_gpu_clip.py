"""The clip kernel at the edges of its layout: a group of eight lanes builds a cell with
one removed vertex, one ring edge and one new vertex per lane, in 32-bit position masks up
to 32 vertices, for at most 37 planes and 48 vertices (64 and 64 in the second round);
beyond each of these another path takes over.  Cells around a point with a given number of
faces, and cuts that remove a given number of vertices at once, cross all of them; every
value has to be the oracle's, bit for bit.
"""
import numpy as np
import pytest

from voronoi_checks import compare

pytestmark = pytest.mark.gpu


def _sphere(n, rng):
    """A cell with about n faces: its generator among n points at nearly one distance."""
    v = rng.normal(size=(n, 3))
    v /= np.linalg.norm(v, axis=1)[:, None]
    return np.concatenate([[[0.5, 0.5, 0.5]], 0.5 + 0.3 * rng.uniform(0.99, 1.01, (n, 1)) * v])


def _prism(n, rng):
    """A cell that is an n-sided prism until its last two neighbours cut off its ends, each
    with all n vertices there (or most of them) at once."""
    a = (np.arange(n) + rng.uniform(-0.2, 0.2, n)) * 2 * np.pi / n
    side = 0.5 + 0.2 * np.stack([np.cos(a), np.sin(a), 0.05 * rng.uniform(-1, 1, n)], 1)
    ends = [[0.5, 0.5, 0.5 + 0.25], [0.51, 0.5, 0.5 - 0.26]]
    return np.concatenate([[[0.5, 0.5, 0.5]], side, ends])


@pytest.mark.parametrize("precision", ["filtered", "fp64"])
@pytest.mark.parametrize("shape,n", [(_prism, n) for n in (5, 7, 8, 9, 15, 16, 17, 30, 33, 40)]
                         + [(_sphere, n) for n in (18, 25, 31, 32, 40, 60, 75)],
                         ids=lambda v: v.__name__[1:] if callable(v) else str(v))
def test_cells_at_the_edges_of_the_layout(gpu_ctx, oracle, shape, n, precision):
    rng = np.random.default_rng(1000 + n)
    g = np.concatenate([shape(n, rng) + [2.0 * k, 0.0, 0.0] for k in range(5)])
    box = ([0, 0, 0], [10, 1, 1])
    orc = oracle.build(g, *box, dim=3, periodic=False)
    gpu = gpu_ctx.build_arrays(g, None, *box, 3, False, precision=precision, pipeline="staged",
                               initial_radius=4.0)
    assert compare(gpu, orc), "expected bit-identical integrals"
    st = gpu_ctx.last_stats()
    fused = gpu_ctx.build_arrays(g, None, *box, 3, False, precision=precision, pipeline="fused")
    assert compare(fused, orc)
    sf = gpu_ctx.last_stats()
    for k in ("cells_built", "neighbours_clipped", "planes_added", "exact_tests", "serial_rings"):
        assert st[k] == sf[k], k


# a generator and its five nearest neighbours in the unit box; the fifth cut removes eight of
# ten vertices, the first ring node among them, and the reference's swaps decide which
# triangle closes that node's fan
SWAPPED = [
    [[0.1316, 0.6167, 0.9615], [0.1312, 0.6156, 0.9756], [0.1306, 0.6206, 0.9465],
     [0.1327, 0.6014, 0.9592], [0.1155, 0.6149, 0.9598], [0.1316, 0.6335, 0.9573]],
    [[0.7081, 0.942, 0.0364], [0.6981, 0.9484, 0.0384], [0.6991, 0.9329, 0.0357],
     [0.7147, 0.9279, 0.0352], [0.714, 0.9469, 0.0221], [0.7074, 0.9432, 0.0527]],
]


@pytest.mark.parametrize("precision", ["filtered", "fp64"])
@pytest.mark.parametrize("case", range(len(SWAPPED)))
def test_ring_start_after_swaps(gpu_ctx, oracle, case, precision):
    rng = np.random.default_rng(case)
    near = np.array(SWAPPED[case])
    v = rng.normal(size=(30, 3))
    ring = near[0] + rng.uniform(0.02, 0.035, (30, 1)) * v / np.linalg.norm(v, axis=1)[:, None]
    g = np.concatenate([near, np.clip(ring, 0.0, 1.0), rng.random((300, 3))])
    orc = oracle.build(g, [0, 0, 0], [1, 1, 1], dim=3, periodic=False, flags=oracle.FACES_ALL | oracle.NO_CSR)
    cells = gpu_ctx.build_cells(g, None, [0, 0, 0], [1, 1, 1], 3, False, precision=precision,
                                pipeline="staged")[0]
    gpu = gpu_ctx.build_arrays(g, None, [0, 0, 0], [1, 1, 1], 3, False, precision=precision, face_mode=1,
                               pipeline="staged")
    assert compare(gpu, orc, faces_all=True)
    assert np.array_equal(cells.cell_centroid, gpu.cell_centroid)
