"""The fused self-matrix build (csrc/ring_kernels.cu): every compile-time order, the run-time
instances at the first and last order of each padded range, upsampled orders other than 2p
(down to p and up to the largest taken) and the first order past them, both layers, against the
oracle's matrices. FP64 sums of some 1e4 terms of one size: 1e-12 relative to the largest entry,
the bound that the build has everywhere else."""
import numpy as np
import pytest

from oracle import sh
from tests.helpers import ellipsoid_pair, rel_err
from ves3d_b200.stokes_velocity import StokesVelocity

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.mark.parametrize("p,p_up", [(2, 4), (3, 6), (4, 8), (5, 10), (6, 12), (6, 6), (6, 13), (7, 9), (8, 16), (8, 15),
                                    (9, 18), (10, 20), (12, 24), (12, 30), (13, 26), (16, 20)])
@pytest.mark.parametrize("single", [True, False])
def test_self_matrix_orders(p, p_up, single):
    X = ellipsoid_pair(p)
    with StokesVelocity(p, p_up) as sv:
        sv.SetSrcCoord(X)
        sv.SetDensitySL(np.zeros(X.size))
        if single:
            M = sv.self_matrix()
        else:
            sv.SetDensityDL(np.zeros(X.size))
            sv()
            M = sv.dl_matrix()
    assert rel_err(M, sh.stokes_singular_matrix(X, p, p_up, single=single)) < TOL


@pytest.mark.parametrize("p,p_up", [(16, 32), (17, 34), (20, 40), (21, 30), (24, 48), (24, 56), (24, 57), (25, 50), (4, 56)])
def test_fused_build_equals_stage_by_stage(p, p_up, monkeypatch):
    """Large orders against the stage-by-stage pipeline (itself checked against the oracle), the
    first unsupported ones included; one vesicle."""
    X = ellipsoid_pair(p)[:3 * sh.ngrid(p)]
    got = []
    for fused in ("1", "0"):
        monkeypatch.setenv("VES3D_FUSED_BUILD", fused)
        with StokesVelocity(p, p_up) as sv:
            sv.SetSrcCoord(X)
            sv.SetDensitySL(np.zeros(X.size))
            sv.SetDensityDL(np.zeros(X.size))
            sv()
            got.append((sv.self_matrix(), sv.dl_matrix()))
    for a, b in zip(*got):
        assert rel_err(a, b) < TOL
