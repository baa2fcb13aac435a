"""Removed regions that have no single ring.  Generators that nearly coincide make cells whose
vertices rounding leaves in contradiction; the reference then finds no triangle that extends
its cycle, and so must the clip kernel, whose walk along the ring's successors leaves the
ring in the cells named here (the region's first node is interior and has no successor).
The error and its cell have to be the oracle's."""
import numpy as np
import pytest

from meshless_voro_b200._native import MvError

pytestmark = pytest.mark.gpu


def _near_duplicates(seed):
    rng = np.random.default_rng(seed)
    n = int(rng.integers(100, 400))
    g = np.round(rng.random((n, 3)) * rng.integers(2, 12)) / 12
    g = g + float(rng.choice([1e-14, 1e-12, 1e-10, 1e-9, 1e-8, 1e-7])) * rng.standard_normal(g.shape)
    return g, bool(rng.integers(0, 2))


# others: generators in a second unit box beside the first, so many that the first round takes
# the tier of 37 planes
@pytest.mark.parametrize("precision", ["filtered", "fp64"])
@pytest.mark.parametrize("seed,cell,others", [
    (22876, 32, 0), (44111, 60, 0), (145642, 77, 0), (20911, 149, 0), (127026, 15, 0),
    (23323, 192, 0), (127873, 72, 0), (127026, 15, 8000), (23323, 192, 8000), (127873, 72, 8000)])
def test_walk_that_leaves_the_ring(gpu_ctx, oracle, seed, cell, others, precision):
    g, periodic = _near_duplicates(seed)
    width = [1, 1, 1]
    if others:
        g = np.concatenate([g, np.random.default_rng(seed).random((others, 3)) + [1, 0, 0]])
        width = [2, 1, 1]
    one = np.zeros(len(g), bool)
    one[cell] = True
    for mask in (one, None):
        orc = oracle.build(g, [0, 0, 0], width, dim=3, periodic=periodic, mask=mask)
        assert orc.status == 3
        with pytest.raises(MvError) as e:
            gpu_ctx.build_arrays(g, mask, [0, 0, 0], width, 3, periodic, precision=precision, pipeline="staged")
        assert (e.value.status, e.value.error_cell) == (orc.status, orc.error_cell)
