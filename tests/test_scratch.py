"""The scratch that a context keeps after calls that return arrays is given back: when
its buffers grow (GPU), and when an allocation is out of memory (the retry, on the CPU)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_allocation_retry(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "alloc_retry_check")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-o", exe, os.path.join(HERE, "native", "alloc_retry_check.cu")], check=True,
                   capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
def test_scratch_goes_when_buffers_grow():
    """Two contexts that end with the buffers of the larger grid: the one that
    extracted the smaller grid before holds no more than the other."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import dmtz_gb300 as dm

    small, large = (96, 96, 96), (100, 100, 100)
    f = np.random.default_rng(1).standard_normal(100 ** 3)
    held, again = [], None
    for extract in (False, True):
        ctx = dm.Context(0)
        ctx.mismatch(f[: 96 ** 3], f[: 96 ** 3], small)  # (what a first call loads stays with the process)
        before = torch.cuda.mem_get_info()[0]
        if extract:
            first = ctx.extract(f[: 96 ** 3], small)
            assert before - torch.cuda.mem_get_info()[0] >= 4 * sum(dm.cell_counts(small))
        ctx.mismatch(f, f, large)
        held.append(before - torch.cuda.mem_get_info()[0])
        if extract:
            again = ctx.extract(f[: 96 ** 3], small)
            assert all(np.array_equal(a, b) for a, b in zip(first, again))
        ctx.close()
    assert held[1] - held[0] < 2 * sum(dm.cell_counts(small)), held
