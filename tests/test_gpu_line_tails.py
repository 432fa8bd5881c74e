"""FP32 line transforms whose last levels share a block between four line
sets: every remainder of levels and of line sets, against dense matrices.

Tolerance: FP32 transforms of two axes, at most six passes that round by 2^-24
of the line's norm each way plus the conversion: 2e-6 relative per level."""
import numpy as np
import pytest

from ps3d_gb300 import Ps3dGpu
from tests.test_fx_transforms import fourier

TOL = 2e-6


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(10, 64, 64), (64, 10, 32), (18, 128, 36), (64, 64, 36), (128, 30, 96), (8, 256, 40)])
def test_mixed_line_operators(shape):
    nx, ny, nz = shape
    g = Ps3dGpu(nx, ny, nz, (0.0, 0.0, 0.0), (2.0, 3.0, 1.0), precision="mixed")
    rng = np.random.default_rng(nx * ny + nz)
    f = rng.standard_normal((nx, ny, nz + 1))
    (fx, ix), (fy, iy) = [[m.astype(np.float64) for m in fourier(n)] for n in (nx, ny)]
    for op, mx, my in (("fftxyp2s", fx, fy), ("fftxys2p", ix, iy)):
        out = getattr(g, op)(f)
        ref = np.einsum("ai,bj,ijk->abk", mx, my, f, optimize=True)
        err = np.sqrt(((out - ref) ** 2).sum((0, 1)) / (ref ** 2).sum((0, 1)))
        assert err.max() < TOL, (op, int(err.argmax()), float(err.max()))
    g.close()
