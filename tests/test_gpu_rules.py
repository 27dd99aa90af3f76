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
