"""Byte ranges of a patch's finishing inputs checked on the host (no GPU): builds
tests/cpp/check_finish_regions.cc with nvcc (host code only) and runs it, past
the node counts whose nodal arrays exceed 4 GB."""
import os
import shutil
import subprocess
import tempfile

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.timeout(600)
def test_finish_regions_on_host():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    with tempfile.TemporaryDirectory() as tmp:
        exe = os.path.join(tmp, "check_finish_regions")
        subprocess.run([nvcc, "-std=c++17", "-O2",
                        "-I", os.path.join(ROOT, "akantu_b200", "csrc"),
                        "-I", os.path.join(ROOT, "include"),
                        "-o", exe, os.path.join(ROOT, "tests", "cpp", "check_finish_regions.cc")],
                       check=True, capture_output=True, text=True)
        out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "fails 0" in out.stdout
