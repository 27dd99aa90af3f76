"""Runs of short rounds that end early or hand a round back, in the host-driven loop and
in the loop graph, against the oracle's loop stopped at the same round: values, edit
counters, rounds."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

FLAGS = (1, 1, 1, 0, 0, 0, 0)


def _correct(ctx, f, g, dims, rel, flags, max_rounds, use_graph):
    """dmtz_correct that also returns an unconverged field and its edit counters."""
    import dmtz_gb300 as dm

    out, cnt = np.array(g, copy=True), np.empty(f.size, np.int32)
    o, r = dm.Opts(*flags, max_rounds, use_graph, 1, 0), dm.Report()
    rc = ctx._L.dmtz_correct(ctx._h, *dims, f.ctypes.data, out.ctypes.data, 0, float(rel), ctypes.byref(o), ctypes.byref(r),
                             cnt.ctypes.data)
    return rc, out, cnt, r.as_dict()


def _same_as_oracle(ctx, f, g, dims, rel, flags, max_rounds, use_graph):
    want, st, wcnt = O.correct(f, g, dims, rel, list(flags), max_outer=500, threads=4, break_stalls=True, max_rounds=max_rounds)
    rc, out, cnt, rep = _correct(ctx, f, g, dims, rel, flags, max_rounds, use_graph)
    # the graph loop does not check the separatrices again once the cap is reached
    unchecked = use_graph and flags[1] and rep["cp_rounds"] + rep["path_rounds"] == max_rounds
    assert rc == (0 if st["converged"] and not unchecked else 4)
    assert np.array_equal(out, want) and np.array_equal(cnt, wcnt)
    assert rep["cp_rounds"] == st["cp_iterations"]
    # (and counts the outer iteration that the cap keeps from starting)
    assert rep["outer_iterations"] == st["outer_iterations"] or (use_graph and rc == 4)
    assert rep["stall_breaks"] == st["stall_breaks"] and rep["initial_mismatch"] == st["initial_mismatch"]
    return st, rep


@pytest.mark.parametrize("use_graph", [0, 1])
@pytest.mark.parametrize("max_rounds", [1, 2, 3, 5, 7, 12])
@pytest.mark.parametrize("dims", [(9, 8, 7), (16, 16, 16), (23, 9, 31)])
def test_round_caps(gpu_ctx, dims, max_rounds, use_graph):
    r = np.random.default_rng(sum(dims))
    V = dims[0] * dims[1] * dims[2]
    x, y, z = np.meshgrid(*[np.linspace(0, 3, n) for n in dims], indexing="ij")
    f = (np.sin(2 * x) * np.cos(3 * y) + 0.3 * np.sin(5 * z) + 0.1 * r.standard_normal(dims)).transpose(2, 1, 0).reshape(-1)
    for rel in (1e-3, 1e-2):
        g = f + rel * (f.max() - f.min()) * r.uniform(-1, 1, V)
        _same_as_oracle(gpu_ctx, f, g, dims, rel, FLAGS, max_rounds, use_graph)


@pytest.mark.parametrize("use_graph", [0, 1])
@pytest.mark.parametrize("flags", [FLAGS, (0, 0, 0, 0, 0, 0, 0)])
@pytest.mark.parametrize("max_rounds", [1, 3])
def test_rounds_handed_back(gpu_ctx, flags, max_rounds, use_graph):
    """Few cells, far apart, so that one round marks more than 160 bricks: the launch ends
    after its update and the repair is done by the kernels it stands for."""
    dims = (96, 96, 96)
    z, y, x = np.meshgrid(*[np.arange(n, dtype=float) for n in dims[::-1]], indexing="ij")
    f = (x + 0.37 * y + 0.11 * z).reshape(-1)
    g = f.copy()
    for i in range(4):
        for j in range(4):
            for k in range(2):
                if (i + j + k) % 4 != 3:  # a new minimum at a brick's corner: its update reaches eight bricks
                    g[(16 + 16 * i) + 96 * ((16 + 16 * j) + 96 * (16 + 32 * k))] -= 1.05
    st, _ = _same_as_oracle(gpu_ctx, f, g, dims, 3.0 / (f.max() - f.min()), flags, max_rounds, use_graph)
    assert st["initial_mismatch"] == [24, 24, 0, 0]
    first = O.correct(f, g, dims, 3.0 / (f.max() - f.min()), list(flags), max_outer=500, threads=4, max_rounds=1)[0]
    v = np.nonzero(first != g)[0]
    marked = set()
    for a, b, c in zip(v % 96, v // 96 % 96, v // 9216):
        marked |= {(p, q, r) for p in {(a - 2) // 8, (a + 1) // 8} for q in {(b - 2) // 4, (b + 1) // 4}
                   for r in {(c - 2) // 4, (c + 1) // 4}}
    assert len(marked) > 160
