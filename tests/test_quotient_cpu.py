"""The quotient of the products' gated epilogue against the division of IEEE 754, on the host (no GPU)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
INC = os.path.join(os.path.dirname(HERE), "blitz_scale_b200", "csrc", "kernels")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_quotient(tmp_path):
    exe = str(tmp_path / "quotient_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", INC, os.path.join(HERE, "native", "quotient_check.cpp"), "-o", exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
