"""kernel_launches of the graph loop: short rounds are one launch among the loop's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [1, 3])
def test_graph_loop_counts_short_rounds(gpu_ctx, seed):
    """8^3 vertices are four bricks, and their few mismatches end in one run of short
    rounds: the loop is that kernel, the repair behind it and a round's end before
    and after.  A correction without a mismatch launches all the rest."""
    dims = (8, 8, 8)
    r = np.random.default_rng(seed)
    z, y, x = np.meshgrid(*[np.arange(n, dtype=float) for n in dims[::-1]], indexing="ij")
    f = (x + 0.37 * y + 0.11 * z).reshape(-1)
    g = f.copy()
    v = int(r.integers(2, 6)) + 8 * (int(r.integers(2, 6)) + 8 * int(r.integers(2, 6)))
    g[v] -= 3.0
    flags = (1, 0, 0, 0, 0, 0, 0)
    _, clean = gpu_ctx.correct(f, f, 0.5, flags, dims=dims, use_graph=1)
    _, rep = gpu_ctx.correct(f, g, 0.5, flags, dims=dims, use_graph=1)
    assert clean["cp_rounds"] == 0 and sum(clean["initial_mismatch"]) == 0
    assert 0 < sum(rep["initial_mismatch"]) <= 32 and 0 < rep["cp_rounds"] < 256 and rep["stall_breaks"] == 0
    assert rep["kernel_launches"] - clean["kernel_launches"] == 4
