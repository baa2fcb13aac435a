"""First neighbour shells at the edges of their search: generators on the faces of the search
grid's cells, boxes far from the origin (where the cell index is rounded most), and radii
that reach the face of a cell; and shells whose 25-bit distance keys collide without being
equal.  Every value has to be the oracle's, bit for bit.
"""
import numpy as np
import pytest

from voronoi_checks import compare

pytestmark = pytest.mark.gpu


def _grid_side(n, dim):
    """Cells per side of the search grid of n generators in a cube (2.2 generators per cell)."""
    return int(np.floor((n / 2.2) ** (1.0 / dim)))


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("anchor,width", [(0.0, 1.0), (1e4, 1.0), (-3e5, 10.0), (700.0, 0.1), (2e14, 1e15)])
@pytest.mark.parametrize("dim", [2, 3])
def test_generators_on_grid_faces(gpu_ctx, oracle, dim, anchor, width, periodic):
    rng = np.random.default_rng(dim)
    n = 900 if dim == 2 else 1500
    side = _grid_side(n, dim)
    u = rng.random((n, dim))
    axis = rng.integers(0, dim, n)  # on a face (or centre plane) of the grid's cells along one axis
    u[np.arange(n), axis] = np.round(2 * side * u[np.arange(n), axis]) / (2.0 * side)
    g = np.zeros((n, 3))
    g[:, :dim] = anchor + np.minimum(u, 1.0 - 1e-12) * width
    box = ([anchor] * 3, [width] * 3)
    orc = oracle.build(g, *box, dim=dim, periodic=periodic)
    gpu = gpu_ctx.build_arrays(g, None, *box, dim, periodic, pipeline="staged")
    assert compare(gpu, orc), "expected bit-identical integrals"


def test_colliding_distance_keys(gpu_ctx, oracle):
    """Neighbours at distances that differ by less than a key's resolution (2^-25 of the
    shell's squared radius), in the opposite order of their indices."""
    rng = np.random.default_rng(5)
    v = rng.normal(size=(24, 3))
    v /= np.linalg.norm(v, axis=1)[:, None]
    r = 0.02 * (1.0 + 1e-10 * np.arange(24)[::-1])
    g = np.concatenate([[[0.5, 0.5, 0.5]], 0.5 + r[:, None] * v, rng.random((6000, 3))])
    orc = oracle.build(g, [0, 0, 0], [1, 1, 1], dim=3, periodic=True)
    for precision in ("filtered", "fp64"):
        gpu = gpu_ctx.build_arrays(g, None, [0, 0, 0], [1, 1, 1], 3, True, precision=precision,
                                   pipeline="staged")
        assert compare(gpu, orc)
