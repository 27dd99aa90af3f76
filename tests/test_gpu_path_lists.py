"""The original field's 2-saddle list after a connectivity check: that check counts
records of decompressed 2-saddles and grows its record arrays alone, so the next
call on the context needs a longer list while its records already fit.  Records
and corrections against the oracle, on a context of its own."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

DIMS = (20, 18, 16)


def _two_saddles(f):
    return int((O.pair(f, DIMS)[2] == -1).sum())


@pytest.mark.parametrize("use_graph", [0, 1])
@pytest.mark.parametrize("strict", [False, True])
def test_two_saddle_list_grows_after_a_connectivity_check(use_graph, strict):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import dmtz_gb300 as dm
    from dmtz_gb300 import synth

    z, y, x = np.meshgrid(*[np.arange(n, dtype=float) for n in DIMS[::-1]], indexing="ij")
    ramp = (x + 0.37 * y + 0.11 * z).reshape(-1)
    noise = np.random.default_rng(3).standard_normal(ramp.size)
    f, g = (a.reshape(-1) for a in synth.make_case("powerlaw", DIMS, 2, 1e-3, "sz"))
    ctx = dm.Context(0)
    try:
        records = len(ctx.path_detect(ramp, noise, DIMS, connectivity=True)[0])
        assert _two_saddles(ramp) < _two_saddles(f) <= records
        got = ctx.path_detect(f, g, DIMS, strict=strict)
        want = O.path_detect(O.pair(f, DIMS), O.pair(g, DIMS), DIMS, strict=strict)[:4]
        assert len(want[0]) > 0
        for a, b in ((0, 1), (2, 3)):
            assert sorted(zip(got[a].tolist(), got[b].tolist())) == sorted(zip(want[a].tolist(), want[b].tolist()))
        flags = (1, 1, 1, 0, 0, 0, 0)
        field, st, cnt = O.correct(f, g, DIMS, 1e-3, list(flags), max_outer=500, break_stalls=True, strict=strict)
        out, rep, gcnt = ctx.correct(f, g, 1e-3, flags, dims=DIMS, use_graph=use_graph, strict=strict, return_counter=True)
        assert st["converged"] and rep["converged"]
        assert np.array_equal(out, field) and np.array_equal(gcnt, cnt)
    finally:
        ctx.close()


@pytest.mark.parametrize("call", ["connectivity", "walls", "correct"])
def test_no_paths_traced_where_none_are_read(call):
    """Connectivity mode and the walls read no traced path: their calls leave no
    room for segments (24 bytes per 16 vertices, 16 per 64) behind."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import dmtz_gb300 as dm

    dims = (176, 176, 176)
    n = dims[0] ** 3
    z, y, x = np.meshgrid(*[np.arange(k, dtype=float) for k in dims[::-1]], indexing="ij")
    f = (x + 0.37 * y + 0.11 * z).reshape(-1)  # few saddles: records and lists are small
    g = f.copy()
    g[n // 2] -= 3e-3 * (f.max() - f.min())
    held = []
    for paths in (False, True):
        ctx = dm.Context(0)
        ctx.mismatch(f, g, dims)
        before = torch.cuda.mem_get_info()[0]
        if not paths and call == "connectivity":
            ctx.path_detect(f, g, dims, connectivity=True)
        elif not paths and call == "walls":
            ctx.wall_detect(f, g, dims)
        elif not paths:
            ctx.correct(f, g, 1e-2, (1, 1, 0, 0, 0, 0, 0), dims=dims)
        elif call == "correct":
            ctx.correct(f, g, 1e-2, (1, 1, 1, 0, 0, 0, 0), dims=dims)
        else:
            ctx.path_detect(f, g, dims)
        held.append(before - torch.cuda.mem_get_info()[0])
        ctx.close()
    room = n // 16 * 24 + n // 64 * 16  # (the arrays per slot may land in memory that is mapped already)
    assert held[0] < room // 2 and held[0] < held[1], held
