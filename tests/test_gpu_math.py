"""The device arithmetic that replaces FP64 instructions (csrc/ck_math.cuh):
conversions between float, double and fixed point exact (ties of the double
result may go either way), exp(-y) and 1 / sqrt within one unit in the last
place, the square root within 0.51 of one, sine and cosine within 2^-59."""

import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
LIMITS = {"widen": 0, "narrow": 0, "sqrt": 0.51, "rsqrt": 1.0, "exp": 1.0, "fixed": 0.5, "sin": 1.0, "cos": 1.0,
          "back": 0.5}


def test_device_arithmetic(tmp_path):
    exe = str(tmp_path / "math_check")
    csrc = os.path.join(HERE, os.pardir, "chimes_calculator_gb300", "csrc")
    subprocess.run(["nvcc", "-std=c++17", "-O2", "-gencode", "arch=compute_103a,code=sm_103a", "-I", csrc,
                    os.path.join(HERE, "math_check.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    got = {ln.split()[0]: float(ln.split()[1]) for ln in out.splitlines()}
    assert set(got) == set(LIMITS)
    for name, limit in LIMITS.items():
        assert got[name] <= limit, (name, got[name])
