"""Application of the self matrices (two columns a lane where rows are even, one where odd;
columns and rows past whole groups) to a density, from the context's own matrix: FP64 sums of at
most 1,872 terms, 1e-13 relative to the largest value, times ten for the transforms around it."""
import numpy as np
import pytest

from oracle import sh
from tests.helpers import rel_err, small_suspension
from ves3d_b200.stokes_velocity import StokesVelocity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,nside", [(2, 1), (3, 2), (4, 2), (5, 1), (7, 2), (8, 1), (12, 2), (13, 1), (16, 1), (24, 1)])
def test_self_apply(p, nside):
    X, f = small_suspension(nside, p, p)
    with StokesVelocity(p) as sv:
        sv.SetSrcCoord(X)
        sv.SetDensitySL(f)
        sv()
        own = sv.parts()[0]
        SL = sv.self_matrix()
    assert rel_err(own, sh.self_apply(SL, f, p)) < 1e-12
