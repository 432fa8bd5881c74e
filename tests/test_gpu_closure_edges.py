"""tcgen05 inference at the ends of its range of levels: columns much shorter
than a tile of 126 rows, and the longest the shared memory takes, whose pitch
nz + 3 is no multiple of the 8 rows of a core matrix.  Held against the warp
engine with the tolerance that the sizes in between have."""
import numpy as np
import pytest

from ps3d_gb300.closure import Closure
from tests.test_gpu_closure import TOL_EMU_OUT, boosted_params, random_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(8, 8, 8), (32, 16, 8), (8, 16, 128)])
def test_engines_agree(dims):
    nx, ny, nz = dims
    vor, vel, _ = random_fields((nx, ny, nz + 1), 5)
    cl = Closure(nx, ny, nz, seed=8)
    cl.set_params(boosted_params(cl))
    cl.scale = 1.0
    assert cl.engine == "tcgen05"
    out = cl.predict(vor, vel)
    cl.check()
    cl.engine = "mma"
    ref = cl.predict(vor, vel)
    assert np.linalg.norm(out - ref) < TOL_EMU_OUT * np.linalg.norm(ref)
    cl.close()
