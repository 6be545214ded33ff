"""The FP64 far field that evaluates each unordered pair once (csrc/far_sym_kernels.cu) and the
small launch shape below it: sizes around the line between them, vesicles that reach over group
borders, coincident points of distinct vesicles, mixed orders, both layers, against the oracle's
direct sums. 20,000 FP64 terms of either sign: 1e-12 relative to the largest value."""
import numpy as np
import pytest

from oracle import sh, stokes
from tests.helpers import rel_err
from ves3d_b200 import _lib, workloads
from ves3d_b200.stokes_velocity import PolydisperseStokesVelocity, StokesVelocity

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _vesicles(n, p, seed):
    side = int(np.ceil(n ** (1.0 / 3.0)))
    X, f = workloads.suspension(side, p, 3.0, semi_axes=(1.0, 1.0, 0.6), deg=4, amp=0.05, seed=seed)
    m = 3 * sh.ngrid(p) * n
    return X[:m].copy(), f[:m].copy()


# 84 points a vesicle at p = 6, 24 at p = 3, 1,200 at p = 24: 7,980 | 8,064 and 7,992 | 8,016 around the
# line at 8,000; 20,328 | 20,496 around the change of block size at 20,480
@pytest.mark.parametrize("n,p", [(1, 6), (2, 3), (95, 6), (96, 6), (333, 3), (334, 3), (15, 16),
                                 (7, 24), (242, 6), (244, 6)])
@pytest.mark.parametrize("dl", [False, True])
def test_far_field_around_the_line(n, p, dl):
    X, f = _vesicles(n, p, 5 + n)
    Xv = X.reshape(n, 3, -1)
    if n > 2:
        Xv[n - 1, :, 4] = Xv[0, :, 3]  # a coincident pair of distinct vesicles counts nothing
    g = np.random.default_rng(n).standard_normal(X.size) if dl else None
    with StokesVelocity(p) as sv:
        sv.SetSrcCoord(X)
        sv.SetDensitySL(f)
        if dl:
            sv.SetDensityDL(g)
        sv()
        far = sv.parts()[1]
    ref = stokes.far_velocity(X, f, p) + (stokes.far_dl_velocity(X, g, p) if dl else 0.0)
    if n == 1:
        assert np.abs(far).max() == 0.0
    else:
        assert rel_err(far, ref) < TOL


def test_paired_sums_equal_the_forced_shapes():
    """One-sided sums (a fixed launch shape) and paired sums of the same points."""
    X, f = _vesicles(18, 16, 3)
    with StokesVelocity(16) as sv:
        sv.SetSrcCoord(X)
        sv.SetDensitySL(f)
        sv()
        a = sv.parts()[1]
        try:
            for waves, nthr in ((4, 256), (16, 384)):
                _lib.set_far_shape(waves, nthr, 2)
                sv.SetDensitySL(f)
                sv()
                assert rel_err(sv.parts()[1], a) < TOL
        finally:
            _lib.set_far_shape(0)


def test_sizes_change_within_one_context():
    """Fewer and more points than the partial sums were sized for, across the line."""
    with StokesVelocity(6) as sv:
        for n in (100, 10, 96, 95, 244, 120):
            X, f = _vesicles(n, 6, n)
            sv.SetSrcCoord(X)
            sv.SetDensitySL(f)
            sv()
            assert rel_err(sv.parts()[1], stokes.far_velocity(X, f, 6)) < TOL


@pytest.mark.parametrize("dl", [False, True])
def test_mixed_orders(dl):
    orders = [4, 6, 16, 3, 12, 7] * 8
    parts = [_vesicles(1, p, 40 + i) for i, p in enumerate(orders)]
    X = np.concatenate([(P[0].reshape(3, -1) + np.array([3.1 * (i % 4), 3.0 * (i // 4 % 4), 3.2 * (i // 16)])[:, None])
                        .reshape(-1) for i, P in enumerate(parts)])
    f = np.concatenate([P[1] for P in parts])
    assert X.size // 3 >= 8000
    g = np.random.default_rng(1).standard_normal(X.size) if dl else None
    with PolydisperseStokesVelocity() as sv:
        sv.SetSrcCoord(X, orders)
        sv.SetDensitySL(f)
        if dl:
            sv.SetDensityDL(g)
        vel = sv()
    assert rel_err(vel, stokes.stokes_velocity_poly(X, f, orders, g)) < TOL
