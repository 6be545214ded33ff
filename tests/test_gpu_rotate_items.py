"""The per-item adjoint rotation in FP64 at each of its orders, with the twelve planes of a rotation
in one CTA (many vesicles) and split over several (few): the same arithmetic, so the same bits, and
the oracle's matrices to 1e-12."""
import numpy as np
import pytest

from oracle import sh
from tests.helpers import rel_err
from ves3d_b200 import workloads
from ves3d_b200.stokes_velocity import StokesVelocity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,n", [(4, 125), (6, 100), (8, 75), (10, 64), (12, 48), (14, 45), (16, 40), (18, 0), (20, 0)])
def test_planes_split_and_whole(p, n):
    X, _ = workloads.suspension(5, p, 3.0, semi_axes=(1.0, 1.0, 0.6), deg=4, amp=0.05, seed=p)
    m = 3 * sh.ngrid(p)
    got = []
    for k in (1, 4, n):  # n: past (p + 1) n = 4 x 148 CTAs (orders 18 and 20 in the few-vesicle form alone)
        if k:
            with StokesVelocity(p) as sv:
                sv.SetSrcCoord(X[:m * k])
                got.append(sv.self_matrix()[0])
    for g in got[1:]:
        assert np.array_equal(g, got[0])
    assert rel_err(got[0], sh.stokes_singular_matrix(X[:m], p, 2 * p)[0]) < 1e-12
