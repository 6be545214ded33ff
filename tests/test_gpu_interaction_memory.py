"""The interaction handle where the partial sums of the paired form find no room on the device: the
one-sided sums, which need none, answer instead (1e-12 of the oracle, as the paired form)."""
import ctypes

import numpy as np
import pytest

from oracle import stokes
from tests.helpers import rel_err
from ves3d_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("with_ctx", [True, False])
def test_no_room_for_partial_sums(with_ctx):
    import torch
    n, few = 60000, 500  # 4 MB of points and values, 58 MB or more of partial sums
    L = ctypes.CDLL(_lib.LIB_PATH)
    slots = L._ZN5ves3d14alltoall_slotsEl
    slots.restype, slots.argtypes = ctypes.c_long, [ctypes.c_long]
    assert 24 * n * slots(n) > 56 * 2 ** 20
    rng = np.random.default_rng(3)
    src, den, pot = rng.standard_normal(3 * n), rng.standard_normal(3 * n), np.full(3 * n, 7.0)
    small = np.zeros(3 * few)
    L = _lib.lib()

    def call(m, out, ctx):
        L.ves3d_stokes_alltoall_f64(src.ctypes.data, den.ctypes.data, m, out.ctypes.data, ctx)

    d = [torch.from_numpy(a).cuda() for a in (src, den)]
    one_sided = torch.zeros(3 * n, dtype=torch.float64, device="cuda")
    _lib.check(L.ves3d_stokes_alltoall_device_f64(d[0].data_ptr(), d[1].data_ptr(), n, one_sided.data_ptr(), None),
               "device")
    ctx = ctypes.c_void_p()
    h = ctypes.byref(ctx) if with_ctx else None
    call(few, small, h)  # kernels loaded, the stream made
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    block = torch.empty(free - 40 * 2 ** 20, dtype=torch.uint8, device="cuda")
    try:
        call(n, pot, h)
    finally:
        del block
        torch.cuda.empty_cache()
    assert np.array_equal(pot, one_sided.cpu().numpy())
    call(n, pot, h)  # with room again
    ref = stokes.alltoall(src[: 3 * few], den[: 3 * few])
    assert rel_err(small, ref) < 1e-12
    assert rel_err(pot, one_sided.cpu().numpy()) < 1e-12
    if with_ctx:
        L.ves3d_interaction_free(ctypes.byref(ctx))
