"""Off-surface targets whose number changes within one context."""
import numpy as np
import pytest

from tests.helpers import small_suspension
from ves3d_b200.stokes_velocity import StokesVelocity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("near", [False, True])
def test_fewer_targets_after_more(near):
    """One context's targets shrink and grow again: every count gives a fresh context's bits. (Fewer
    targets split the sources over more segments than more targets do.)"""
    p = 12
    X, f = small_suspension(3, p, 22)
    T = np.random.default_rng(9).uniform(-2.0, 8.0, (20000, 3))

    def values(sv, counts):
        sv.SetSrcCoord(X)
        sv.SetDensitySL(f)
        sv.set_near_singular(near)
        out = []
        for m in counts:
            sv.SetTrgCoord(T[:m])
            out.append(sv.eval_targets())
        return out

    counts = [20000, 9472, 50, 9472, 20000]
    with StokesVelocity(p) as sv:
        got = values(sv, counts)
    for m, u in zip(counts[:3], got):
        with StokesVelocity(p) as sv:
            assert np.array_equal(u, values(sv, [m])[0])
    assert np.array_equal(got[3], got[1]) and np.array_equal(got[4], got[0])
