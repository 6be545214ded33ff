"""Transforms and builds of several orders called from several threads at once: every call is answered,
with the bits that it has alone. (A kernel's shared-memory limit belongs to the kernel, not to the launch.)"""
import threading

import numpy as np
import pytest

from oracle import sh
from tests.helpers import small_suspension
from ves3d_b200.stokes_velocity import SHTrans, StokesVelocity

pytestmark = pytest.mark.gpu


def _together(jobs):
    errors, gate = [], threading.Barrier(len(jobs))

    def run(job):
        try:
            gate.wait()
            job()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=run, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:2]


def test_transforms_of_two_orders():
    import torch

    def job(p, seed):
        st = torch.cuda.Stream()
        t = SHTrans(p, stream=st.cuda_stream)
        X = torch.from_numpy(np.random.default_rng(seed).standard_normal(2 * sh.ngrid(p))).cuda()
        S, ref = (torch.zeros(2 * sh.ncoef(p), dtype=torch.float64, device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        t.forward(X, ref)
        torch.cuda.synchronize()

        def loop():
            for _ in range(3000):
                t.forward(X, S)
            assert torch.equal(S, ref)
        return loop

    _together([job(p, i) for i, p in enumerate((5, 32, 9, 32))])


def test_builds_of_several_orders():
    def job(p, q, seed):
        X, f = small_suspension(1, p, seed)
        sv = StokesVelocity(p, q)

        def one():
            sv.SetSrcCoord(X)
            sv.SetDensitySL(f)
            return sv()
        ref = one()

        def loop():
            for _ in range(300):
                assert np.array_equal(one(), ref)
            sv.close()
        return loop

    _together([job(p, q, i) for i, (p, q) in enumerate(((9, 18), (12, 30), (9, 19), (12, 18)))])
