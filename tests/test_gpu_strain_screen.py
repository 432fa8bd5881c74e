"""adapt's reductions of the FP64 form (screened strain maxima, per-column
sums) against the oracle's full Jacobi sweeps, over field magnitudes down to
where the FP32 screen cannot order points and every point is swept.

Tolerance: strains and sums of O(1e4) products, each a few FP64 units off
after the transforms (2e-15 per field, tests of the transforms): 1e-11
relative leaves three decades."""
import numpy as np
import pytest

import oracle
from ps3d_gb300 import Ps3dGpu, ic

TOL = 1e-11


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1e-11, 1e-4, 1.0, 1e6])
@pytest.mark.parametrize("shape", [(16, 12, 32), (12, 16, 30), (8, 10, 64), (32, 8, 8)])
def test_reductions_match_the_oracle(shape, scale):
    nx, ny, nz = shape
    lo, ex = ic.BELTRAMI_BOX["lower"], ic.BELTRAMI_BOX["extent"]
    vor, pert = ic.beltrami_plus_perturbation(nx, ny, nz, seed=nx)
    g = Ps3dGpu(nx, ny, nz, lo, ex, cflmax=0.5)
    o = oracle.Oracle(nx, ny, nz, lo, ex, cflmax=0.5)
    for s in (g, o):
        s.setup_fields(scale * vor, scale * pert)
    _, dg = g.advance(0.0)
    _, do = o.advance(0.0)
    for k in ("ggmax", "usggmax", "lsggmax", "vorch", "ke", "en", "vortmax", "umax", "vmax", "wmax"):
        assert abs(dg[k] - do[k]) <= TOL * abs(do[k]) + 1e-300, (k, dg[k], do[k])
    g.close()
