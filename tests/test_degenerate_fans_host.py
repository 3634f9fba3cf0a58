"""Fans of elements that name a node twice (a mesh the model refuses, once it is
planned): builds tests/cpp/check_degenerate_fans.cc against akb_patch_build.cu
with nvcc (host code only) and the address sanitizer, and runs it."""
import os
import shutil
import subprocess
import tempfile

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.timeout(600)
def test_degenerate_fans_on_host():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    with tempfile.TemporaryDirectory() as tmp:
        exe = os.path.join(tmp, "check_degenerate_fans")
        subprocess.run([nvcc, "-std=c++17", "-O1", "-g", "-Xcompiler", "-fsanitize=address",
                        "-I", os.path.join(ROOT, "akantu_b200", "csrc"),
                        "-I", os.path.join(ROOT, "include"), "-o", exe,
                        os.path.join(ROOT, "tests", "cpp", "check_degenerate_fans.cc"),
                        os.path.join(ROOT, "akantu_b200", "csrc", "akb_patch_build.cu")],
                       check=True, capture_output=True, text=True)
        out = subprocess.run([exe], capture_output=True, text=True,
                             env=dict(os.environ, ASAN_OPTIONS="detect_leaks=0"))
    assert out.returncode == 0, out.stdout + out.stderr
    assert "fails 0" in out.stdout
