"""One critical-point fix round against the oracle at list lengths where the
kernel gives a warp 1, 2, 4, ... 32 cells."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(6, 5, 4), (15, 14, 12), (19, 17, 16), (25, 24, 20), (33, 30, 28), (50, 47, 45)])
@pytest.mark.parametrize("edit_type", [0, 1])
def test_fix_round_matches_oracle(gpu_ctx, dims, edit_type):
    r = np.random.default_rng(sum(dims))
    V = dims[0] * dims[1] * dims[2]
    f = r.standard_normal(V)
    rng = float(f.max() - f.min())
    rel = 0.02
    g = f + rel * rng * r.uniform(-1, 1, V)
    cnt = r.integers(1, 6, V).astype(np.int32)
    P, Q = O.pair(f, dims, 4), O.pair(g, dims, 4)
    want, _ = O.fix_cp(f, g, cnt, rng * rel, rng, edit_type, 1, P, Q, O.cp_mismatch(P, Q, dims), dims)
    got = gpu_ctx.fix_round(f, g, cnt, rel, 1, edit_type, dims)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("dims", [(9, 8, 7), (16, 16, 16), (23, 9, 31), (40, 33, 12)])
@pytest.mark.parametrize("rel", [1e-3, 1e-2])
@pytest.mark.parametrize("max_rounds", [0, 7])
def test_short_rounds_match_oracle(gpu_ctx, dims, rel, max_rounds):
    """The host-driven loop, whose rounds of short lists run back to back on the
    device, against the oracle's loop: values, edit counters, rounds, also where a
    round cap ends them early."""
    import dmtz_gb300 as dm

    r = np.random.default_rng(sum(dims) + int(rel * 1e4))
    V = dims[0] * dims[1] * dims[2]
    x, y, z = np.meshgrid(*[np.linspace(0, 3, n) for n in dims], indexing="ij")
    f = (np.sin(2 * x) * np.cos(3 * y) + 0.3 * np.sin(5 * z) + 0.1 * r.standard_normal(dims)).transpose(2, 1, 0).reshape(-1)
    g = f + rel * (f.max() - f.min()) * r.uniform(-1, 1, V)
    flags = (1, 1, 1, 0, 0, 0, 0)
    want, st, wcnt = O.correct(f, g, dims, rel, list(flags), max_outer=500, threads=4, break_stalls=True, max_rounds=max_rounds)
    if not st["converged"]:
        with pytest.raises(dm.DmtzError):
            gpu_ctx.correct(f, g, rel, flags, dims=dims, max_rounds=max_rounds)
        return
    out, rep, cnt = gpu_ctx.correct(f, g, rel, flags, dims=dims, return_counter=True, max_rounds=max_rounds)
    assert np.array_equal(np.asarray(out).reshape(-1), want) and np.array_equal(np.asarray(cnt).reshape(-1), wcnt)
    assert rep["cp_rounds"] == st["cp_iterations"] and rep["outer_iterations"] == st["outer_iterations"]
    assert rep["stall_breaks"] == st["stall_breaks"]
