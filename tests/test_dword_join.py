"""dw_join_int (csrc/dword.cuh), by which the mixed mode reads its split matrix: the bits of the FP64
sum of the pair, compiled as host code."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "sayram-2d_gb300", "csrc")


# around the edges of the integer path (hi below 2^-63, the float range's top), the usual range, and the
# exponents at which a part of the pair is subnormal, zero or infinite
@pytest.mark.parametrize("lo_e,hi_e", [(-66, -60), (-59, 60), (120, 130), (-160, -67), (-1074, -900), (1000, 1023)])
def test_join_gives_the_bits_of_the_sum(tmp_path, lo_e, hi_e):
    cxx = shutil.which("g++")
    cuda_inc = "/usr/local/cuda/include"
    if not cxx or not os.path.isdir(cuda_inc):
        pytest.skip("g++ or the CUDA headers are missing")
    exe = str(tmp_path / "join_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-I", cuda_inc,
                    os.path.join(HERE, "dword", "join_check.cc"), "-o", exe], check=True)
    out = subprocess.run([exe, str(lo_e), str(hi_e)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
