"""RotateAll at the ends of its range of orders, odd and even, with remainders of its groups of
longitudes (four at a time, two at p = 24 and 25) and with the longitudes of a rotation in one CTA
(many fields) and split over several (few), against the oracle: 1e-12 relative to the largest value."""
import numpy as np
import pytest

from oracle import sh
from tests.helpers import rel_err
from ves3d_b200._lib import Ves3dError
from ves3d_b200.stokes_velocity import SHTrans

pytestmark = pytest.mark.gpu


def _rotate(p, S):
    import torch
    out = torch.zeros(S.size // (p * (p + 2)) * (p + 1) * p * p * (p + 2), dtype=torch.float64, device="cuda")
    SHTrans(p).RotateAll(torch.from_numpy(S).cuda(), out)
    return out.cpu().numpy()


@pytest.mark.parametrize("p", [2, 3, 4, 5, 7, 10, 16, 23, 24, 25])
def test_orders(p):
    S = np.random.default_rng(p).standard_normal(3 * 2 * p * (p + 2))
    assert rel_err(_rotate(p, S), sh.rotate_all(S, p, 3)) < 1e-12


@pytest.mark.parametrize("p", [3, 6, 13])
def test_few_and_many(p):
    S = np.random.default_rng(p).standard_normal((120, 3 * p * (p + 2)))
    many = _rotate(p, S.reshape(-1)).reshape(120, -1)
    assert np.array_equal(many[7], _rotate(p, S[7].copy()))


def test_too_large_an_order_is_an_error():
    with pytest.raises(Ves3dError):
        _rotate(26, np.zeros(3 * 26 * 28))
