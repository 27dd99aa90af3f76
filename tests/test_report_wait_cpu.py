"""The host's wait for a round's counts (report_wait.cuh), compiled for the host: a
stream that ends without having written them is an error, not a round."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_report_wait(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "report_wait_check")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-o", exe, os.path.join(HERE, "native", "report_wait_check.cu")], check=True,
                   capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
