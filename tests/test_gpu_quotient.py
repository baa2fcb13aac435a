"""quotients (mv_geom.cuh) gives correctly rounded quotients wherever it accepts its operands:
compared bit for bit with IEEE division on the host, over mantissas drawn at random and near
the hard cases (next to one and two, few bits set), exponents over the whole range, and
zeros, subnormals, infinities and NaN on either side, which it has to refuse.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from meshless_voro_b200 import build as B

SOURCE = """
#include "mv_geom.cuh"
__global__ void k(const double* a, const double* b, double* q, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  mv::D3 r;
  // the other two components are always acceptable
  q[i] = mv::quotients(mv::D3{3.0, a[i], -0.7}, b[i], &r) ? r.y : __longlong_as_double(-1);
}
extern "C" int quotients(const double* a, const double* b, double* q, int n) {
  double *da, *db, *dq;
  const size_t m = 8 * (size_t)n;
  if (cudaMalloc(&da, m) || cudaMalloc(&db, m) || cudaMalloc(&dq, m)) return 1;
  cudaMemcpy(da, a, m, cudaMemcpyHostToDevice);
  cudaMemcpy(db, b, m, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(da, db, dq, n);
  const int e = (int)cudaMemcpy(q, dq, m, cudaMemcpyDeviceToHost);
  cudaFree(da), cudaFree(db), cudaFree(dq);
  return e;
}
"""


def _operands(n, rng):
    kind = rng.integers(0, 4, n)
    one, bits = np.uint64(1), np.uint64((1 << 52) - 1)
    mant = rng.integers(0, 1 << 52, n).astype(np.uint64)
    few = rng.integers(0, 16, n).astype(np.uint64)
    mant = np.where(kind == 1, few, mant)                   # next to 1
    mant = np.where(kind == 2, bits - few, mant)            # next to 2
    mant = np.where(kind == 3, (one << rng.integers(0, 52, n).astype(np.uint64)), mant)
    expo = np.where(rng.random(n) < 0.7, rng.integers(1023 - 60, 1023 + 60, n),
                    rng.integers(0, 2048, n)).astype(np.uint64)
    sign = rng.integers(0, 2, n).astype(np.uint64) << np.uint64(63)
    return (sign | (expo << np.uint64(52)) | mant).view(np.float64)


@pytest.mark.gpu
def test_divisor_is_correctly_rounded(tmp_path):
    src, lib = tmp_path / "q.cu", tmp_path / "q.so"
    src.write_text(SOURCE)
    subprocess.run([B.NVCC, *B.NVCC_FLAGS, "-I", B.CSRC, "-shared", str(src), "-o", str(lib)], check=True)
    fn = ctypes.CDLL(os.fspath(lib)).quotients
    rng = np.random.default_rng(17)
    special = np.array([0.0, -0.0, 1.0, -1.0, 3.0, np.inf, -np.inf, np.nan, 5e-324, 2.0 ** -1022,
                        2.0 ** 400, 2.0 ** -400, 2.0 ** 1023])
    a = np.concatenate([_operands(4_000_000, rng), np.repeat(special, len(special))])
    b = np.concatenate([_operands(4_000_000, rng), np.tile(special, len(special))])
    q = np.empty_like(a)
    p = lambda v: v.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    assert fn(p(a), p(b), p(q), len(a)) == 0
    with np.errstate(all="ignore"):
        want = a / b
    refused = q.view(np.int64) == -1
    inside = [(np.abs(v) >= 2.0 ** -400) & (np.abs(v) < 2.0 ** 400) for v in (a, b)]
    assert np.array_equal(refused, ~(inside[0] & inside[1]))
    assert np.array_equal(q.view(np.uint64)[~refused], want.view(np.uint64)[~refused])
    assert (~refused).sum() > 1_000_000
