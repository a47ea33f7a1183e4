"""The fit's division by a shared reciprocal on the CPU: tests/fit_division.cu
built for the host."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_shared_reciprocal_gives_the_quotient(tmp_path):
    if shutil.which("nvcc") is None:
        pytest.skip("no nvcc")
    exe = str(tmp_path / "fit_division")
    subprocess.check_call(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "--fmad=false", "-std=c++17",
                           "-Xcompiler", "-ffp-contract=off", "-o", exe, os.path.join(ROOT, "tests", "fit_division.cu")])
    p = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout[-2000:]
