"""The fused step's fan records checked on the host (no GPU): builds
tests/cpp/check_fan_layout.cc against akantu_b200/csrc/akb_patch_build.cu with
nvcc (host code only) and runs it, on structured and scrambled tetrahedral and
triangular meshes, stars, tiny caps, forced interface nodes, nodes of no
element and a degenerate element."""
import os
import shutil
import subprocess
import tempfile

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.timeout(600)
def test_fan_records_on_host():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    with tempfile.TemporaryDirectory() as tmp:
        exe = os.path.join(tmp, "check_fan_layout")
        subprocess.run([nvcc, "-std=c++17", "-O2",
                        "-I", os.path.join(ROOT, "akantu_b200", "csrc"),
                        "-I", os.path.join(ROOT, "include"),
                        "-o", exe, os.path.join(ROOT, "tests", "cpp", "check_fan_layout.cc"),
                        os.path.join(ROOT, "akantu_b200", "csrc", "akb_patch_build.cu")],
                       check=True, capture_output=True, text=True)
        out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "fails 0" in out.stdout
