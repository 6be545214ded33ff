"""Device memory of the far field's partial sums: a mixed context holds the 32 sets that its FP32 sums
write, not the FP64 form's (up to 80), until FP64 sums run; a graph captured before them stays valid."""
import ctypes

import numpy as np
import pytest

from tests.helpers import small_suspension
from ves3d_b200 import _lib
from ves3d_b200.stokes_velocity import PolydisperseStokesVelocity, StokesVelocity

pytestmark = pytest.mark.gpu


def _used():
    import torch
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


@pytest.mark.parametrize("poly", [False, True])
def test_mixed_partial_sums(poly):
    p, nside = 4, 9  # 29,160 points, 0.7 MB a set; the two forms' contexts differ in nothing else
    nv = nside ** 3
    X, f = small_suspension(nside, p, 92)
    L = ctypes.CDLL(_lib.LIB_PATH)
    sets = L._ZN5ves3d9far_slotsEl  # of the FP64 form
    sets.restype, sets.argtypes = ctypes.c_long, [ctypes.c_long]
    more = (sets(X.size // 3) - 32) * 8 * X.size
    assert more > 20e6
    orders = np.full(nv, p)

    def memory(prec):
        base = _used()
        with PolydisperseStokesVelocity(prec) if poly else StokesVelocity(p, precision=prec) as sv:
            sv.SetSrcCoord(*((X, orders) if poly else (X,)))
            sv.SetDensitySL(f)
            sv()
            return _used() - base

    for prec in ("fp64", "mixed"):  # modules loaded
        memory(prec)
    assert abs(memory("fp64") - memory("mixed") - more) <= 2 ** 22  # allocations are whole blocks of 2 MB


def test_graph_outlives_fp64_sums():
    """FP64 sums of an implicit step get a buffer beside the one that a captured evaluation holds."""
    p = 6
    X, f = small_suspension(2, p, 93)
    with StokesVelocity(p, precision="mixed") as sv:
        sv.SetSrcCoord(X)
        sv.SetDensitySL(f)
        sv.set_implicit_params(0.01, 0.05, 1.0)
        sv.capture_eval()
        sv.SetDensitySL(f)
        sv.launch_eval_graph()
        ref = sv.parts()
        sv.implicit_solve(tol=1e-6, max_iter=20)
        sv.SetDensitySL(f)
        sv.launch_eval_graph()
        for a, b in zip(sv.parts(), ref):
            assert np.array_equal(a, b)
