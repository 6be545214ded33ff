"""The near-singular kernel's quotient by a shared divisor has the bits of the division, over 2^28 numerators
and divisors of its range (built here with nvcc against the kernels' header)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _build(tmp_path):
    from ves3d_b200 import build
    exe = str(tmp_path / "quotient_test")
    flags = [f for f in build.NVCC_FLAGS if f not in ("-shared", "-Xcompiler", "-fPIC")]
    subprocess.check_call([build._nvcc(), *flags, "-I", build.CSRC, "-o", exe,
                           os.path.join(ROOT, "tests", "cpp", "quotient_test.cu")])
    return exe


@pytest.mark.gpu
def test_quotient_equals_division(tmp_path):
    out = subprocess.run([_build(tmp_path)], capture_output=True, text=True, check=True).stdout.split()
    assert out == [str(2 ** 28), "0"]
