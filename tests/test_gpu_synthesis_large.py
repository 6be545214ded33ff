"""Synthesis at orders whose rows fill shared memory: where rows padded to whole groups of four latitudes
no longer fit, unpadded ones are taken. Against the oracle, to 2e-11 of the largest value: the transforms'
1e-12 at order 33, times four for the longer recurrences of the tables and four for the longer sums."""
import numpy as np
import pytest

from oracle import sh
from tests.helpers import rel_err
from ves3d_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,p1,grads", [(52, 123, True), (52, 124, True), (53, 120, True), (53, 121, True),
                                        (64, 96, True), (96, 100, False), (98, 96, False), (85, 124, False)])
def test_synthesis_large(p, p1, grads):
    import torch
    nf = 3
    S = np.random.default_rng(p + p1).standard_normal(nf * sh.ncoef(p))
    dS = torch.from_numpy(S).cuda()
    ref = sh.shc2grid(S, p, p1, grads=True)
    outs = [torch.zeros(nf * sh.ngrid(p1), dtype=torch.float64, device="cuda") for _ in range(3)]
    ptrs = [o.data_ptr() if grads or i == 0 else None for i, o in enumerate(outs)]
    _lib.check(_lib.lib().ves3d_sht_backward(dS.data_ptr(), nf, p, p1, *ptrs, None), "bwd")
    for o, r, q in zip(outs, ref, ptrs):
        assert q is None or rel_err(o.cpu().numpy(), r) < 2e-11
