"""Rounds that re-pair the whole grid, and rounds with as many cells that do not: a grid of
8192 bricks (the smallest that is ever re-paired whole) with noise everywhere, whose first
rounds reach most bricks, and with noise in an eighth of it, whose first round alone is
taken whole.  Values, edit counters and rounds against the oracle's loop stopped at the
same round, in both loops."""
import functools

import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_short_rounds import FLAGS, _correct

pytestmark = pytest.mark.gpu

DIMS = (128, 64, 128)
BRICKS = 16 * 16 * 32
REL = 1e-2


@functools.lru_cache(maxsize=None)
def _field(everywhere):
    W, H, D = DIMS
    z, y, x = np.meshgrid(*[np.arange(n, dtype=float) for n in DIMS[::-1]], indexing="ij")
    f = (x + 0.37 * y + 0.11 * z).reshape(-1)
    noise = np.random.default_rng(5).uniform(-1, 1, f.size).reshape(D, H, W)
    if not everywhere:
        noise[64:] = 0
        noise[:, 32:] = 0
        noise[:, :, 64:] = 0
    return f, f + REL * (f.max() - f.min()) * noise.reshape(-1)


@functools.lru_cache(maxsize=None)
def _oracle(everywhere, flags, max_rounds):
    f, g = _field(everywhere)
    return O.correct(f, g, DIMS, REL, list(flags), max_outer=500, threads=4, break_stalls=True, max_rounds=max_rounds)


@pytest.mark.parametrize("use_graph", [0, 1])
@pytest.mark.parametrize("flags", [FLAGS, (0, 0, 0, 0, 0, 0, 0)])
@pytest.mark.parametrize("everywhere", [True, False])
def test_first_rounds(gpu_ctx, everywhere, flags, use_graph):
    f, g = _field(everywhere)
    want, st, wcnt = _oracle(everywhere, flags, 3)
    assert sum(st["initial_mismatch"][0:4:1 if flags[0] else 3]) >= BRICKS // 2 and not st["converged"]
    # the first round's update reaches anchors 2 below to 1 above
    v = np.nonzero(_oracle(everywhere, flags, 1)[0] != g)[0]
    a, b, c = v % DIMS[0], v // DIMS[0] % DIMS[1], v // (DIMS[0] * DIMS[1])
    marked = np.zeros((32, 16, 16), bool)
    for dx in (-2, 1):
        for dy in (-2, 1):
            for dz in (-2, 1):
                marked[np.clip(c + dz, 0, 127) // 4, np.clip(b + dy, 0, 63) // 4, np.clip(a + dx, 0, 127) // 8] = True
    assert (marked.sum() >= BRICKS // 2) == everywhere
    rc, out, cnt, rep = _correct(gpu_ctx, f, g, DIMS, REL, flags, 3, use_graph)
    assert rc == 4 and rep["cp_rounds"] == st["cp_iterations"] == 3
    assert np.array_equal(out, want) and np.array_equal(cnt, wcnt)
    assert rep["initial_mismatch"] == st["initial_mismatch"] and rep["stall_breaks"] == st["stall_breaks"]
