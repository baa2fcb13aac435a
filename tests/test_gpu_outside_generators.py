"""Generators outside the box.  The search grid keeps them in the cells at its walls, so a
query has to look there although its ball ends beyond the wall.  In a periodic box they are
ordinary generators (a program that moves its generators and wraps them afterwards has
such); in a closed one their cells are what the reference's arithmetic makes of them.  Every
value has to be the oracle's (which here enumerates all images), bit for bit, in each of the
pipelines."""
import numpy as np
import pytest

from meshless_voro_b200._native import MvError
from test_zz_no_alloc import noalloc_build

pytestmark = pytest.mark.gpu
BOX = ([0, 0, 0], [1, 1, 1])
N = {1: 300, 2: 700, 3: 1000}
KEYS = {"cell_volume": "volume", "cell_centroid": "centroid", "cell_safety_radius": "safety_radius",
        "face_left": "face_left", "face_right": "face_right", "face_area": "face_area",
        "face_centroid": "face_centroid", "face_normal": "face_normal", "face_shift_code": "face_shift_code",
        "cell_face_offset": "face_offset", "cell_face_count": "face_count",
        "cell_face_connections": "cell_face_connections"}


def _same(got, orc):
    for k, o in KEYS.items():
        assert np.array_equal(got[k] if isinstance(got, dict) else getattr(got, k), getattr(orc, o)), k


def _build(gpu_ctx, route, g, mask, dim, periodic, precision):
    if route == "batch":
        job = dict(generators=g, anchor=BOX[0], width=BOX[1], dimensionality=dim, periodic=periodic, mask=mask)
        inside = dict(job, generators=g - np.floor(g), mask=None)
        return gpu_ctx.build_batch([inside, job], precision=precision)[1]
    if route == "noalloc":
        return noalloc_build(pytest.importorskip("torch"), g, *BOX, dim, periodic, precision, mask)
    return gpu_ctx.build_arrays(g, mask, *BOX, dim, periodic, precision=precision, pipeline=route)


def _cells_per_side(n, dim):
    return int(np.floor((n / 2.2) ** (1.0 / dim)))


@pytest.mark.parametrize("precision", ["filtered", "fp64"])
@pytest.mark.parametrize("route", ["staged", "fused", "batch", "noalloc"])
@pytest.mark.parametrize("clump", [False, True])
@pytest.mark.parametrize("cells", [0.2, 0.9, 1.7, 3.2])
@pytest.mark.parametrize("dim", [1, 2, 3])
def test_periodic(gpu_ctx, oracle, dim, cells, clump, route, precision):
    rng = np.random.default_rng(dim)
    n = N[dim]
    reach = cells / _cells_per_side(n, dim)
    g = rng.random((n, 3))
    for a in range(dim):  # half of those near a wall cross it
        low, high = g[:, a] < reach, g[:, a] > 1.0 - reach
        cross = rng.random(n) < 0.5
        g[low & cross, a] += 1.0
        g[high & cross, a] -= 1.0
    if clump:  # so dense that its cells' first shells are much thinner than the way to the box
        centre = rng.random(3)
        centre[rng.integers(0, dim)] = 1.0 + reach
        g = np.concatenate([g, centre + 0.02 * reach * rng.standard_normal((80, 3))])
    g[:, dim:] = 0.0
    orc = oracle.build(g, *BOX, dim=dim, periodic=True, flags=oracle.BRUTE_FORCE)
    assert orc.status == 0
    _same(_build(gpu_ctx, route, g, None, dim, True, precision), orc)


@pytest.mark.parametrize("route", ["staged", "fused", "batch", "noalloc"])
@pytest.mark.parametrize("dim,seed", [(d, s) for d in (1, 2, 3) for s in range(6)])
def test_closed(gpu_ctx, oracle, dim, seed, route):
    """Outside by a fraction of a box width to several, along one axis to all."""
    rng = np.random.default_rng(seed)
    g = rng.random(((0, 12, 60, 300)[dim], 3))
    g[:, dim:] = 0.0
    for i in range(3):
        for a in rng.permutation(dim)[:rng.integers(1, dim + 1)]:
            d = (0.2, 0.9, 3.5)[i] * rng.uniform(0.5, 1.5)
            g[i, a] = rng.choice([-d, 1.0 + d])
    for i in range(4):  # one at a time, so that an error is that cell's; then those inside
        mask = np.arange(len(g)) == i if i < 3 else np.arange(len(g)) >= 3
        orc = oracle.build(g, *BOX, dim=dim, periodic=False, mask=mask, flags=oracle.BRUTE_FORCE)
        if orc.status == 0:
            _same(_build(gpu_ctx, route, g, mask, dim, False, "filtered"), orc)
        else:
            with pytest.raises(MvError) as e:
                _build(gpu_ctx, route, g, mask, dim, False, "filtered")
            assert e.value.status == orc.status
