"""The folded Grid2SHC (csrc/grid2shc_kernels.cu) at each order it is instantiated for and the
general kernel at those beside them, through the application of the self matrices (three
functions a vesicle, so counts that leave remainders) and through the build (9 nc a vesicle),
against the oracle and against the general kernel: 1e-12 relative to the largest value."""
import numpy as np
import pytest

from oracle import sh
from tests.helpers import ellipsoid_pair, rel_err
from ves3d_b200.stokes_velocity import StokesVelocity

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.mark.parametrize("p", [3, 4, 6, 8, 10, 12, 14, 16, 18, 20, 22, 24])
@pytest.mark.parametrize("nves", [1, 2])
def test_folded_against_general_and_oracle(p, nves, monkeypatch):
    X = ellipsoid_pair(p)[:3 * nves * sh.ngrid(p)]
    f = np.random.default_rng(p).standard_normal(X.size)
    got = []
    for folded in ("1", "0"):
        monkeypatch.setenv("VES3D_TC_ANALYSIS", folded)
        with StokesVelocity(p) as sv:
            sv.SetSrcCoord(X)
            sv.SetDensitySL(f)
            sv()
            got.append((sv.self_matrix(), sv.parts()[0]))
    assert rel_err(got[0][0], got[1][0]) < TOL
    assert rel_err(got[0][1], got[1][1]) < TOL
    assert rel_err(got[0][1], sh.self_apply(got[0][0], f, p)) < TOL
