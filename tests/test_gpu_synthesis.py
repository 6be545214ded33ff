"""Synthesis with derivatives at function counts and latitude counts that leave remainders in
its groups of functions and of four latitudes, and with the derivative outputs left out, against
the oracle: 1e-12 relative to the largest value, as the transforms have elsewhere."""
import numpy as np
import pytest

from oracle import sh
from tests.helpers import rel_err
from ves3d_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,p1", [(2, 2), (3, 7), (6, 12), (7, 7), (12, 12), (16, 16), (16, 33), (24, 48), (33, 33)])
@pytest.mark.parametrize("nf", [1, 2, 3, 9])
def test_synthesis_remainders(p, p1, nf):
    import torch
    S = np.random.default_rng(p1 + nf).standard_normal(nf * sh.ncoef(p))
    dS = torch.from_numpy(S).cuda()
    ref = sh.shc2grid(S, p, p1, grads=True)
    outs = [torch.zeros(nf * sh.ngrid(p1), dtype=torch.float64, device="cuda") for _ in range(3)]
    L = _lib.lib()
    _lib.check(L.ves3d_sht_backward(dS.data_ptr(), nf, p, p1, *[o.data_ptr() for o in outs], None), "bwd")
    for o, r in zip(outs, ref):
        assert rel_err(o.cpu().numpy(), r) < 1e-12
    outs[0].zero_()
    _lib.check(L.ves3d_sht_backward(dS.data_ptr(), nf, p, p1, outs[0].data_ptr(), None, None, None), "values alone")
    assert rel_err(outs[0].cpu().numpy(), ref[0]) < 1e-12
