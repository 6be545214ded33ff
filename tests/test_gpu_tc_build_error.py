"""A tensor-core build that reports an incomplete result: with several order groups queued at once the
failed group's matrices alone are given up, whichever group it is, and the next evaluation rebuilds them.
The error word is set from the host."""
import ctypes

import numpy as np
import pytest

from tests.helpers import small_suspension
from ves3d_b200 import _lib
from ves3d_b200._lib import Ves3dError
from ves3d_b200.stokes_velocity import PolydisperseStokesVelocity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("failed", [0, 2])
def test_failed_group_of_two(failed):
    runs = [(16, 2), (8, 3), (16, 2)]
    orders = np.concatenate([np.full(n, p) for p, n in runs])
    parts, parts2, dens = [], [], []
    for i, (p, n) in enumerate(runs):
        X, f = small_suspension(2, p, 60 + i)
        X = X.reshape(8, 3, -1)[:n] + 12.0 * i
        parts.append(X.reshape(-1))
        parts2.append((1.01 * X).reshape(-1))
        dens.append(f.reshape(8, -1)[:n].reshape(-1))
    X, X2, f = (np.concatenate(a) for a in (parts, parts2, dens))
    hook = _lib.lib().ves3d_svp_test_build_error
    hook.restype, hook.argtypes = ctypes.c_int, [ctypes.c_void_p, ctypes.c_int, ctypes.c_int]
    with PolydisperseStokesVelocity("mixed") as sv:
        sv.SetSrcCoord(X2, orders)
        sv.SetDensitySL(f)
        ref = sv()
        sv.SetSrcCoord(X, orders)
        sv.SetDensitySL(f)
        sv()
        sv.SetSrcCoord(X2, orders)
        sv.SetDensitySL(f)
        hook(sv._h, failed, 1)
        with pytest.raises(Ves3dError, match="bounded wait"):
            sv()
        assert [hook(sv._h, r, 0) for r in range(3)] == [int(r != failed) for r in range(3)]
        assert np.array_equal(sv(), ref)
        assert [hook(sv._h, r, 0) for r in range(3)] == [1, 1, 1]
