"""The FP64 form's sums are compensated term by term: helicity terms of
+-2^60 at two levels of a column cancel, and what is left are the ones in
between.  An accumulator that rounds at 2^60 loses all of those; the
compensated one keeps each, so the sum is exact."""
import ctypes

import numpy as np
import pytest

from ps3d_gb300 import _lib
from tests.test_zz_no_alloc import _cudart, _noalloc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(8, 8, 128), (6, 10, 270), (3, 5, 1024)])
def test_small_terms_between_large_ones_count(shape):
    nx, ny, nz = shape
    vel = np.ones((3, nx, ny, nz + 1))
    vor = np.zeros_like(vel)
    vor[0] = 1.0
    vor[0, ..., 3] = 2.0 ** 60  # levels of one lane, 1 + (nz - 64) / 32 ones between them
    vor[0, ..., 3 + (nz - 32) // 32 * 32] = -2.0 ** 60
    ones = float(nx * ny * (nz + 1 - 2 - 1))  # two large values, the end levels by half
    rt, L = _cudart(), _lib.lib()
    out = ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(out), ctypes.c_size_t(24)) == 0
    ptrs = [out]
    try:
        got = _noalloc(rt, L, vel, vor, nx, ny, nz, nz + 1, None, out, ptrs)
        assert got[2] * (nx * ny * nz) == pytest.approx(ones, rel=4 * 2.0 ** -53)  # the two products with 1 / cells
    finally:
        for p in ptrs:
            rt.cudaFree(p)
