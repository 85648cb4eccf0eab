"""The quotient of the mixture weights and the bottom solve's beta (csrc/ae_div.h), compiled with g++ and
compared with a / d over random and edge operands (tests/cpp/div_by_check.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_div_by(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "div_by_check")
    # -ffp-contract=off: only the operations written as fma are fused, as in the device code
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                    "-I", os.path.join(ROOT, "anisotropicfracture_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "div_by_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
