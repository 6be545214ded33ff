"""All-pairs sums (the interaction handle) and sums at off-surface targets at the edges of their
tiles, segments and of the paired form's range, against the oracle's direct sums: FP64 sums of up
to 2e4 terms, 1e-12 relative to the largest value."""
import ctypes

import numpy as np
import pytest

from oracle import stokes
from tests.helpers import rel_err, small_suspension
from ves3d_b200 import _lib
from ves3d_b200.stokes_velocity import StokesVelocity

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.mark.parametrize("n", [2, 63, 64, 65, 255, 257, 3999, 4000, 4001, 9217, 20480, 20481])
def test_interaction_sizes(n):
    rng = np.random.default_rng(n)
    src, den = rng.standard_normal(3 * n), rng.standard_normal(3 * n)
    src[3 * (n - 1):] = src[:3]  # a coincident pair counts nothing
    ref = stokes.alltoall(src, den)
    L, ctx, pot = _lib.lib(), ctypes.c_void_p(), np.full(3 * n, 7.0)
    for m in (n, max(2, n // 2), n):  # the handle's work space is kept for fewer points
        L.ves3d_stokes_alltoall_f64(src.ctypes.data, den.ctypes.data, m, pot.ctypes.data, ctypes.byref(ctx))
    L.ves3d_interaction_free(ctypes.byref(ctx))
    if n == 2:
        assert np.all(pot == 0.0)
    else:
        assert rel_err(pot, ref) < TOL
    import torch
    d = [torch.from_numpy(a).cuda() for a in (src, den)]
    out = torch.zeros(3 * n, dtype=torch.float64, device="cuda")
    _lib.check(L.ves3d_stokes_alltoall_device_f64(d[0].data_ptr(), d[1].data_ptr(), n, out.data_ptr(), None), "device")
    torch.cuda.synchronize()
    assert np.all(out.cpu().numpy() == 0.0) if n == 2 else rel_err(out.cpu().numpy(), ref) < TOL


@pytest.mark.parametrize("m", [1, 63, 64, 65, 4736, 4737, 9601])
@pytest.mark.parametrize("dl", [False, True])
def test_target_sizes(m, dl):
    p = 5
    X, f = small_suspension(2, p, 21)
    rng = np.random.default_rng(m)
    g = rng.standard_normal(X.size) if dl else None
    T = rng.uniform(-3.0, 6.0, (m, 3))
    with StokesVelocity(p) as sv:
        sv.SetSrcCoord(X)
        sv.SetDensitySL(f)
        if dl:
            sv.SetDensityDL(g)
        sv.SetTrgCoord(T)
        u = sv.eval_targets()
    assert rel_err(u, stokes.target_velocity(X, f, p, T, g)) < TOL
