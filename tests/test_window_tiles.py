"""Which residual-window tiles a decode launch fetches (host arithmetic of the kernel's own rule)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc not available")
def test_tiles_without_rows_are_left_out(tmp_path):
    exe = tmp_path / "window_check"
    subprocess.run([NVCC, "-O2", "-std=c++17", "-Wno-deprecated-gpu-targets", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "r2omni_b200", "csrc"), "-o", str(exe), os.path.join(ROOT, "tests", "window_check.cu")],
                   check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("OK"), out.stdout
