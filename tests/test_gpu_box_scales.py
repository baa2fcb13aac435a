"""Boxes far from unit size, where squared distances leave the range in which f32 has its
full precision (or vanish, or overflow), and boxes whose sides differ by many orders of
magnitude.  Every value has to be the oracle's, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SCALES = [1e-14, 1e-15, 3e-16, 1e-18, 1e-20, 1e-22, 1e-23, 1e-24, 1e-30, 1e17, 3e18, 1e19, 1e25]
UNEVEN = [[1.0, 1e-9, 1e-20], [1e-3, 1e-18, 1e-22], [1e-17, 1e-15, 3e-16], [1e18, 1e19, 3e19]]


@pytest.mark.parametrize("pipeline", ["staged", "fused"])
@pytest.mark.parametrize("precision", ["filtered", "fp64"])
@pytest.mark.parametrize("width,dim,periodic",
                         [([s] * 3, d, p) for s in SCALES for d in (2, 3) for p in (False, True)]
                         + [(w, 3, False) for w in UNEVEN])
def test_box_scales(gpu_ctx, oracle, width, dim, periodic, precision, pipeline):
    g = np.random.default_rng(3).random((400, 3)) * width
    g[:, dim:] = 0.0
    box = ([0.0] * 3, width)
    orc = oracle.build(g, *box, dim=dim, periodic=periodic)
    assert orc.status == 0
    gpu = gpu_ctx.build_arrays(g, None, *box, dim, periodic, precision=precision, pipeline=pipeline)
    for a, b in [(gpu.cell_volume, orc.volume), (gpu.cell_centroid, orc.centroid),
                 (gpu.cell_safety_radius, orc.safety_radius), (gpu.face_left, orc.face_left),
                 (gpu.face_right, orc.face_right), (gpu.face_shift_code, orc.face_shift_code),
                 (gpu.face_area, orc.face_area), (gpu.face_centroid, orc.face_centroid),
                 (gpu.face_normal, orc.face_normal), (gpu.cell_face_offset, orc.face_offset),
                 (gpu.cell_face_count, orc.face_count),
                 (gpu.cell_face_connections, orc.cell_face_connections)]:
        assert np.array_equal(a, b)
