"""The order of separatrix records (record_sort.h), compiled for the host: as std::sort's,
for no record, ties in the first column, ids of any size."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_record_sort(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "record_sort_check")
    subprocess.run([cxx, "-std=c++17", "-O2", "-o", exe, os.path.join(HERE, "native", "record_sort_check.cpp")], check=True,
                   capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
