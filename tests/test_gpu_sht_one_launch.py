"""The one-launch transforms and filters (csrc/sht_fused_kernels.cu) over their range of orders,
odd ones and both ends included, one past it, with function counts that leave remainders, against
the oracle: 1e-12 relative to the largest value."""
import numpy as np
import pytest

from oracle import sh
from tests.helpers import rel_err
from ves3d_b200 import _lib
from ves3d_b200.stokes_velocity import SHTrans

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.mark.parametrize("p", [2, 3, 4, 5, 7, 8, 12, 15, 16, 17, 24, 31, 32, 33])
@pytest.mark.parametrize("nf", [1, 2, 5])
def test_transforms(p, nf):
    import torch
    rng = np.random.default_rng(100 * p + nf)
    X, S = rng.standard_normal(nf * sh.ngrid(p)), rng.standard_normal(nf * sh.ncoef(p))
    dX, dS = torch.from_numpy(X).cuda(), torch.from_numpy(S).cuda()
    oS, oX, oF = torch.zeros_like(dS), torch.zeros_like(dX), torch.zeros_like(dX)
    t = SHTrans(p, filter_freq=max(1, p // 2))
    t.forward(dX, oS)
    assert rel_err(oS.cpu().numpy(), sh.grid2shc(X, p, p)) < TOL
    t.backward(dS, oX)
    assert rel_err(oX.cpu().numpy(), sh.shc2grid(S, p, p)) < TOL
    ref = sh.low_pass(X, p, max(1, p // 2))
    t.lowPassFilter(dX, oF)
    assert rel_err(oF.cpu().numpy(), ref) < TOL
    t.lowPassFilter(dX, dX)  # in place
    assert torch.equal(dX, oF)


def test_many_functions():
    """More functions than one round of CTAs holds."""
    import torch
    p, nf = 6, 20011
    X = np.random.default_rng(0).standard_normal((nf, sh.ngrid(p)))
    X[-1] = X[0]
    out = torch.zeros(nf * sh.ncoef(p), dtype=torch.float64, device="cuda")
    SHTrans(p).forward(torch.from_numpy(X.reshape(-1)).cuda(), out)
    o = out.cpu().numpy().reshape(nf, -1)
    pick = [0, 1, 777, 10000, nf - 2, nf - 1]
    assert rel_err(o[pick].reshape(-1), sh.grid2shc(X[pick].reshape(-1), p, p)) < TOL
    assert np.array_equal(o[0], o[-1])
