"""The kernel probe brackets every column transform of the FP64 form: the
launches of a right-hand side and the fields they read and write, in the fused
kernels (up to 512 levels) and in the separate ones beyond."""
import pytest

from ps3d_gb300 import Ps3dGpu, ic

pytestmark = pytest.mark.gpu
COLUMNS = 3


@pytest.mark.parametrize("shape, vor2vel, source", [
    # combine + difference + decomposition of one component (3 fields), two
    # combines (4), w and dw/dz (4); the tendency from five products (8)
    ((16, 12, 32), (3, 11), (1, 8)),
    # combine, decomposition, two combines, dct and dst, two fields each; three decompositions
    ((8, 10, 540), (6, 12), (3, 6)),
])
def test_column_launches_and_bytes(shape, vor2vel, source):
    nx, ny, nz = shape
    g = Ps3dGpu(nx, ny, nz, ic.BELTRAMI_BOX["lower"], ic.BELTRAMI_BOX["extent"])
    g.setup_fields(*ic.beltrami_plus_perturbation(nx, ny, nz, seed=1))
    field = 8.0 * nx * ny * (nz + 1)
    for call, (launches, fields) in ((g.vor2vel, vor2vel), (g.source, source)):
        g.probe(COLUMNS)
        call()
        ms, n, nbytes = g.probe_result()
        assert (n, nbytes) == (launches, fields * field) and ms > 0.0, call
    g.probe(0)
    g.close()
