"""The kernels' own FP64 reciprocal and quotient, the preconditioner's conversions and the double-word
reciprocal as the device forms it, against CUDA's operations: every exponent of the divisor, both signs,
powers of two, the exponents where the code branches, subnormals, zeros, infinities and NaN."""
import os
import subprocess

import pytest

from sayram2d_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))

# one unit in the last place of a result rounded correctly (what the third-order series and one residual
# step leave); the same bits wherever the plain operators are taken and in the conversions; in units of
# 2^-48, the square of the 2 ulp that CUDA documents for __fdividef (16) and two roundings of 2^-22 to FP32 (4
# each)
BOUNDS = {"rcp64_ulp": 1, "div64_ulp": 1, "rcp64_special": 0, "div64_special": 0, "narrow": 0, "widen": 0, "dw_rcp": 24}


@pytest.mark.gpu
def test_against_the_plain_operations(tmp_path):
    exe = str(tmp_path / "quotient_check")
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-ffp-contract=off", "-I", build.CSRC,
                    os.path.join(HERE, "dword", "quotient_check.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    worst = {ln.split()[0]: float(ln.split()[1]) for ln in out.strip().splitlines()}
    assert set(worst) == set(BOUNDS)
    for k, b in BOUNDS.items():
        assert worst[k] <= b, (k, worst)
