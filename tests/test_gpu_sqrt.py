"""The integer-pipe square root (epic_gb300/csrc/fix_math.cuh) equals the binary64 one bit for bit: 2e9
roots covering every seed, rounding boundaries and special operands (tests/cuda/sqrt_check.cu, compiled
here with nvcc)."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "epic_gb300", "csrc")


def test_integer_square_root_is_the_root(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "sqrt_check")
    subprocess.run([nvcc, "-O3", "-std=c++17", "-fmad=false", "-gencode", "arch=compute_103a,code=sm_103a", "-I", CSRC, "-o", exe,
                    os.path.join(HERE, "cuda", "sqrt_check.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr
