"""Near-singular target evaluations of a context whose upsampling order changes: the sources at p_up, their
latitudes and weights follow the order, so every evaluation has a fresh context's bits."""
import numpy as np
import pytest

from tests.helpers import small_suspension
from ves3d_b200.stokes_velocity import StokesVelocity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dl", [False, True])
def test_order_up_raised_and_lowered(dl):
    p = 8
    X, f = small_suspension(2, p, 41)
    rng = np.random.default_rng(4)
    g = rng.standard_normal(X.size)
    T = rng.uniform(-1.5, 4.5, (200, 3))

    def fill(sv):
        sv.SetSrcCoord(X)
        sv.SetDensitySL(f)
        if dl:
            sv.SetDensityDL(g)
        sv.set_near_singular(True)
        sv.SetTrgCoord(T)

    orders = [16, 27, 12, 16]
    with StokesVelocity(p, orders[0]) as sv:
        fill(sv)
        got = [sv.eval_targets()]
        n_near = sv.near_info()
        for q in orders[1:]:
            sv.set_order_up(q)
            assert sv.near_info() == n_near  # the last evaluation's, until the next one
            got.append(sv.eval_targets())
            n_near = sv.near_info()
    for q, u in zip(orders, got):
        with StokesVelocity(p, q) as sv:
            fill(sv)
            assert np.array_equal(u, sv.eval_targets())
