"""Device memory of a context with a double layer: the fused build of either layer needs the rotated
coefficients, their contraction and the self-matrix grid (21 MB a vesicle at p = 16), not the stage
buffers of the build without it (96 MB a vesicle more)."""
import numpy as np
import pytest

from tests.helpers import small_suspension
from ves3d_b200.stokes_velocity import StokesVelocity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dl_first", [False, True])
def test_double_layer_scratch(dl_first):
    import torch
    p, nv = 16, 8
    X, f = small_suspension(2, p, 91)

    def used():
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free

    with StokesVelocity(p) as warm:  # modules loaded, context memory taken
        warm.SetSrcCoord(X[: X.size // nv])
        warm.SetDensitySL(f[: f.size // nv])
        warm.SetDensityDL(f[: f.size // nv])
        warm()
    base = used()
    with StokesVelocity(p) as sv:
        sv.SetSrcCoord(X)
        sv.SetDensitySL(f)
        if not dl_first:
            sv()
        sv.SetDensityDL(np.ones_like(f))
        sv()
        # scratch, two sets of self matrices of 6 MB a vesicle, and fields
        assert used() - base < nv * 45e6
