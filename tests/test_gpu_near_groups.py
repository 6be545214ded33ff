"""Near-singular correction over both group widths (orders to 15 share a warp, larger ones take
one each) and at the ends of their ranges, several near vesicles per target and none, against the
oracle (the correction's 1e-10), and the error of a target near too many vesicles."""
import numpy as np
import pytest

from oracle import near, sh, stokes
from tests.helpers import rel_err, small_suspension
from ves3d_b200._lib import Ves3dError
from ves3d_b200.stokes_velocity import StokesVelocity

pytestmark = pytest.mark.gpu


def _off_surface(X, p, rng, n, dists):
    ng = sh.ngrid(p)
    Xv, nrm = X.reshape(-1, 3, ng), stokes.unit_normal(X, p).reshape(-1, 3, ng)
    out = []
    for i in range(n):
        v, k = rng.integers(Xv.shape[0]), rng.integers(ng)
        out.append(Xv[v, :, k] + dists[i % len(dists)] * (1 if i % 2 == 0 else -1) * nrm[v, :, k])
    return np.array(out)


@pytest.mark.parametrize("p,n", [(4, 33), (15, 3), (16, 3), (17, 2)])
@pytest.mark.parametrize("dl", [False, True])
def test_orders(p, n, dl):
    nside = 2 if p < 8 else 1
    X, f = small_suspension(nside, p, 31, spacing=2.4)
    rng = np.random.default_rng(p)
    g = rng.standard_normal(X.size) if dl else None
    T = np.concatenate([_off_surface(X, p, rng, n, [0.05, 0.1, 0.3]), rng.uniform(8.0, 9.0, (2, 3))])
    with StokesVelocity(p) as sv:
        sv.SetSrcCoord(X)
        sv.SetDensitySL(f)
        if dl:
            sv.SetDensityDL(g)
        SL = sv.self_matrix()
        sv()
        DL = sv.dl_matrix() if dl else None
        sv.SetTrgCoord(T)
        sv.set_near_singular(True)
        u = sv.eval_targets().reshape(-1, 3)
        r_near, n_near = sv.near_info()
    ref, info = near.target_velocity_near(X, f, p, T, g=g, SL=SL, DL=DL, return_info=True)
    assert n_near == len(info["pairs"]) and abs(r_near - info["r_near"]) < 1e-13 * r_near
    assert rel_err(u, ref) < 1e-10


def test_too_many_near_vesicles_is_an_error():
    p = 6
    X, f = small_suspension(2, p, 3, spacing=0.05)  # eight vesicles on top of each other
    T = np.concatenate([np.full((40, 3), 30.0), X.reshape(-1, 3, sh.ngrid(p))[0, :, :3].T + 1e-3])
    with StokesVelocity(p) as sv:
        sv.SetSrcCoord(X)
        sv.SetDensitySL(f)
        sv.SetTrgCoord(T)
        sv.set_near_singular(True)
        with pytest.raises(Ves3dError, match="target 40 "):
            sv.eval_targets()
        sv.SetTrgCoord(T[:40])  # the context goes on
        assert np.isfinite(sv.eval_targets()).all()
