"""The rounds that follow the first in builds without dense cells: cells beside voids (the
wide round's shell, and what even that does not close) and cells with more vertices than
the staged tiers hold (handed to the large tier), against the oracle."""
import numpy as np
import pytest

from meshless_voro_b200._native import MvError
from voronoi_checks import compare

pytestmark = pytest.mark.gpu
BOX = ([0, 0, 0], [1, 1, 1])


def _check(gpu_ctx, oracle, g, dim, periodic, precision):
    """The build's statistics; None where the oracle (as the reference) gives up on a cell,
    and the build has to name the same cell and reason."""
    orc = oracle.build(g, *BOX, dim=dim, periodic=periodic)
    if orc.status != 0:
        with pytest.raises(MvError) as e:
            gpu_ctx.build_arrays(g, None, *BOX, dim, periodic, precision=precision, pipeline="staged")
        assert (e.value.status, e.value.error_cell) == (orc.status, orc.error_cell)
        return None
    v = gpu_ctx.build_arrays(g, None, *BOX, dim, periodic, precision=precision, pipeline="staged")
    assert compare(v, orc)
    return gpu_ctx.last_stats()


@pytest.mark.parametrize("precision", ["filtered", "fp64"])
@pytest.mark.parametrize("radius", [0.12, 0.2, 0.3, 0.42])
@pytest.mark.parametrize("dim", [2, 3])
def test_voids(gpu_ctx, oracle, dim, radius, precision):
    rng = np.random.default_rng(int(100 * radius))
    g = rng.random((4000, 3))
    g[:, dim:] = 0.0
    r = np.sqrt((((g - 0.5) * (np.arange(3) < dim)) ** 2).sum(axis=1))
    st = _check(gpu_ctx, oracle, g[r > radius], dim, True, precision)
    assert st["staged_wide"] > 0


@pytest.mark.parametrize("precision", ["filtered", "fp64"])
@pytest.mark.parametrize("stars", [1, 3, 24])
def test_many_faced_cells(gpu_ctx, oracle, stars, precision):
    """Generators at the centres of spheres of 90 others: cells of about 90 faces."""
    rng = np.random.default_rng(stars)
    side = 3
    c = (np.stack(np.meshgrid(*[np.arange(side)] * 3), -1).reshape(-1, 3)[:stars] + 0.5) / side
    c += 0.01 * rng.random(c.shape)
    g = rng.random((2000, 3))
    g = g[np.sqrt(((g[:, None] - c[None]) ** 2).sum(-1)).min(axis=1) > 0.16]
    v = rng.normal(size=(stars, 90, 3))
    v /= np.linalg.norm(v, axis=2)[:, :, None]
    g = np.concatenate([g, c, (c[:, None] + 0.14 * v).reshape(-1, 3)])
    st = _check(gpu_ctx, oracle, rng.permutation(g), 3, False, precision)
    assert st is None or st["overflow_cells"] >= stars


@pytest.mark.parametrize("precision", ["filtered", "fp64"])
@pytest.mark.parametrize("n", [800, 7103, 7104, 7105, 9000, 24_000])
@pytest.mark.parametrize("periodic", [False, True])
def test_tier_of_the_first_round(gpu_ctx, oracle, n, periodic, precision):
    """Around the size up to which the first round takes the wide tier: Poisson cells, and a
    cell of some 40 faces, which only the wide tier holds."""
    rng = np.random.default_rng(n)
    v = rng.normal(size=(44, 3))
    v /= np.linalg.norm(v, axis=1)[:, None]
    c = np.array([0.4, 0.5, 0.6])
    r = 1.6 * n ** (-1.0 / 3.0)
    g = rng.random((2 * n, 3))
    g = g[np.sqrt(((g - c) ** 2).sum(axis=1)) > 1.15 * r][: n - 45]
    g = rng.permutation(np.concatenate([g, [c], c + r * (1.0 + 0.03 * rng.random((44, 1))) * v]))
    assert len(g) == n
    _check(gpu_ctx, oracle, g, 3, periodic, precision)
