"""The constant twiddles of the register DFTs (cmblensing_b200/csrc/lf_fft.cuh), on the CPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not found")
def test_constant_twiddles(tmp_path):
    """Closer than rounding the two parts (0.5 each): with the better of the two factored forms the worst angle of
    the 32-point transform, pi/8, is 0.373 units of 2^-24 off.  The double constants are held in double: one unit
    each for the argument, the quotient and the product."""
    exe = tmp_path / "twiddle_check"
    subprocess.check_call(["nvcc", "-std=c++17", "-Wno-deprecated-gpu-targets", "-gencode",
                           "arch=compute_100a,code=sm_100a", "-o", str(exe),
                           os.path.join(HERE, "native", "twiddle_check.cu")])
    r = subprocess.run([str(exe), "0.374"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert float(r.stdout.split()[3]) < 3.0
