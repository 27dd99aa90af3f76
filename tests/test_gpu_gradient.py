"""The gradient kernels at the edges of their tiles: grids around the march's
32 x 16 columns and its planes per block, thin grids with long axes, the brick
kernel's last grid and the march's first, against the oracle's five passes; and
the gradient after a repair around scattered changes.  Whole numbers: equality."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# bricks of 8 x 4 x 4: up to 3 per SM (456 on 152 SMs) take the brick kernel
MARCH = [(32, 16, 90), (33, 17, 91), (31, 15, 88), (64, 48, 41), (65, 49, 37), (2, 2, 2100), (1200, 5, 4), (3, 1100, 3),
         (34, 18, 130)]
BRICK = [(8, 4, 4), (9, 5, 5), (7, 3, 2), (2, 2, 2), (31, 33, 40)]


@pytest.mark.parametrize("kind", ["normal", "ties"])
@pytest.mark.parametrize("dims", MARCH + BRICK)
def test_full_gradient(gpu_ctx, dims, kind):
    from oracle import oracle as O

    n = dims[0] * dims[1] * dims[2]
    r = np.random.default_rng(n)
    f = r.standard_normal(n) if kind == "normal" else r.integers(0, 4, n).astype(np.float64)
    for got, want, name in zip(gpu_ctx.extract(f, dims), O.pair(f, dims, threads=4), ("PV", "PE", "PF", "PT")):
        assert np.array_equal(got, want), name


@pytest.mark.parametrize("shape", [0, 1, 2])
@pytest.mark.parametrize("dims", [(17, 9, 9), (40, 23, 70)])
def test_repaired_gradient(gpu_ctx, dims, shape):
    """A correction's repairs (brick lists of every shape, host loop and graph)
    end in the oracle's field: every round's lists come from repaired bricks."""
    from dmtz_gb300 import synth
    from oracle import oracle as O

    f, g = synth.make_case("powerlaw", dims, 5, 1e-2, "sz")
    f, g = f.reshape(-1), g.reshape(-1)
    flags = (1, 1, 1, 0, 0, 0, 0)
    want, _, _ = O.correct(f, g, dims, 1e-2, list(flags), break_stalls=True)
    saved = gpu_ctx.get_tuning()
    try:
        gpu_ctx.set_tuning(shape, 16)
        for graph in (0, 1):
            out, rep = gpu_ctx.correct(f, g, 1e-2, flags, dims=dims, use_graph=graph)
            assert rep["converged"] and np.array_equal(out, want)
    finally:
        gpu_ctx.set_tuning(*saved)
