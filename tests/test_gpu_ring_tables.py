"""The FP64 build's tables in a mixed context at p = 16, whose own builds run on the tensor cores: made when
an FP64 build first needs them (a double layer, an implicit step, another upsampling order)."""
import numpy as np
import pytest

from tests.helpers import small_suspension
from ves3d_b200.stokes_velocity import StokesVelocity

pytestmark = pytest.mark.gpu


def test_fp64_builds_of_a_mixed_context():
    p = 16
    X, f = small_suspension(1, p, 94)

    def matrices(prec, q):
        with StokesVelocity(p, q, precision=prec) as sv:
            sv.SetSrcCoord(X)
            sv.SetDensitySL(f)
            sv.SetDensityDL(f)
            return sv.self_matrix(), sv.dl_matrix()

    SL, DL = matrices("fp64", 32)
    SL30 = matrices("fp64", 30)[0]
    with StokesVelocity(p, precision="mixed") as sv:
        sv.SetSrcCoord(X)
        sv.SetDensitySL(f)
        sv()
        sv.SetDensityDL(f)
        assert np.array_equal(sv.dl_matrix(), DL)
        sv.set_implicit_params(0.01, 0.05, 1.0)
        assert np.array_equal(sv.self_matrix(), SL)
        sv.set_order_up(30)
        assert np.array_equal(sv.self_matrix(), SL30)
        sv.set_order_up(32)
        assert np.array_equal(sv.self_matrix(), SL)
