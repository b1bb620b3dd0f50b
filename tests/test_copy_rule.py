"""Which device-to-device copies run as a kernel (no GPU): those between a field
and plain memory of the handle's own GPU while that GPU is current."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_copy_rule(tmp_path):
    exe = str(tmp_path / "copy_rule")
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(CUDA, "include"),
                    os.path.join(HERE, "cpp", "copy_rule.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
