"""An evaluation queues its stages without waiting between them: the times of the stages, values
read back at once, replaced inputs and replaced surfaces are those of a call that waits, and the
surface operations agree whether or not something is queued before them."""
import numpy as np
import pytest

from oracle import stokes
from tests.helpers import rel_err, small_suspension
from ves3d_b200.stokes_velocity import StokesVelocity

pytestmark = pytest.mark.gpu


def test_queued_evaluations_and_times():
    import torch
    p = 8
    X, f = small_suspension(2, p, 11)
    X2, f2 = small_suspension(2, p, 12)
    with StokesVelocity(p) as sv:
        sv.SetSrcCoord(X)
        sv.SetDensitySL(f)
        v = sv()
        t = sv.stage_times()
        assert all(x > 0 for x in t.values())
        assert rel_err(v, stokes.stokes_velocity_sl(X, f, p)) < 1e-12
        # device input that is overwritten as soon as the call has returned
        dX, df = torch.from_numpy(X2).cuda(), torch.from_numpy(f2).cuda()
        sv.SetSrcCoord(dX)
        dX.fill_(7.0)
        sv.SetDensitySL(df)
        torch.cuda.synchronize()
        out = torch.empty_like(df)
        sv(out)
        assert rel_err(out.cpu().numpy(), stokes.stokes_velocity_sl(X2, f2, p)) < 1e-12
        # the double layer's build and far field have times of their own
        sv.SetDensityDL(f)
        sv()
        assert sv.far_dl_ms() > 0


def test_surface_ops_after_queued_work():
    p = 6
    X, f = small_suspension(2, p, 3)
    with StokesVelocity(p) as a, StokesVelocity(p) as b:
        for sv in (a, b):
            sv.SetSrcCoord(X)
            sv.set_implicit_params(0.01, 0.05, 1.0)
        a.SetDensitySL(f)
        a()
        for op, n in enumerate((0, 1, 3, 3, 3, 0, 1, 4, 0, 3)):  # values per point of the operand
            arg = np.resize(f, n * f.size // 3) if n else None
            u, w = a.surface_op(op, arg), b.surface_op(op, arg)
            assert np.array_equal(u, w) and np.isfinite(u).all()
            assert np.array_equal(a.surface_op(op, arg), u)


def test_another_stream_after_the_surfaces():
    """A stream set after SetSrcCoord finds the surfaces' fields formed."""
    import torch
    p = 16
    X, f = small_suspension(4, p, 21)
    with StokesVelocity(p) as sv:
        sv.SetSrcCoord(X)
        sv.SetDensitySL(f)
        ref = sv()
    streams = [torch.cuda.Stream() for _ in range(2)]
    dX, df = torch.from_numpy(X).cuda(), torch.from_numpy(f).cuda()
    torch.cuda.synchronize()
    with StokesVelocity(p) as sv:
        for i in range(6):
            sv.set_stream(streams[i % 2].cuda_stream)
            sv.SetSrcCoord(dX)
            sv.set_stream(streams[1 - i % 2].cuda_stream)
            sv.SetDensitySL(df)
            assert np.array_equal(sv(), ref)
        sv.set_stream(None)
