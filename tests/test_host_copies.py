"""mv_copy_arrays: copies and widenings of result arrays, at the sizes where its blocks and
threads begin and end; refused arguments."""
import ctypes as C

import numpy as np
import pytest

from meshless_voro_b200 import _native as N

BLOCK = 1 << 16


@pytest.mark.parametrize("n", [0, 1, BLOCK - 1, BLOCK, BLOCK + 1, 5 * BLOCK + 3, 1_500_000])
def test_copies_and_widenings(n):
    rng = np.random.default_rng(n)
    src = [(rng.random(n), np.float64), (rng.integers(-2 ** 31, 2 ** 31, n).astype(np.int32), np.int64),
           (rng.integers(0, 256, n).astype(np.uint8), np.int32), (rng.integers(0, 9, n).astype(np.int32), np.int32),
           (rng.integers(0, 2 ** 62, n), np.int64), (rng.integers(0, 256, n).astype(np.uint8), np.uint8)]
    copies = N.ArrayCopies()
    got = [copies.take(C.c_void_p(s.ctypes.data), n, s.itemsize, t) for s, t in src]
    copies.run()
    for (s, t), g in zip(src, got):
        assert g.dtype == t and np.array_equal(g, s.astype(t))
        assert not np.shares_memory(g, s)


def test_nothing_to_copy_and_refusals():
    lib = N.lib()
    assert lib.mv_copy_arrays(None, 0) == N.MV_OK
    a = np.zeros(4)
    for bad in ((a.ctypes.data, a.ctypes.data, 4, 0, 0), (a.ctypes.data, a.ctypes.data, 4, 6, 0),
                (a.ctypes.data, a.ctypes.data, -1, 3, 0), (None, a.ctypes.data, 1, 3, 0)):
        assert lib.mv_copy_arrays((N.Copy * 1)(bad), 1) == N.MV_ERR_ARG
    assert lib.mv_copy_arrays(None, 1) == N.MV_ERR_ARG
