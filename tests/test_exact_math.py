"""The branch-free quotients and square roots of the linearisation (rgbd-flow_b200/csrc/exact_math.cuh) equal the FP32
operators bit for bit, over every mantissa (tests/cpp/exact_math_check.cu)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.gpu
@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc to compile the check")
def test_quotients_and_roots_equal_the_operators(tmp_path):
    exe = str(tmp_path / "exact_math_check")
    subprocess.run(["nvcc", "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe,
                    os.path.join(HERE, "cpp", "exact_math_check.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "no error different 0", r.stdout + r.stderr
