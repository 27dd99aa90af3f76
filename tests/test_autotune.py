"""The autotuner: what its cache accepts, and that measuring leaves the inputs and
degenerate inputs alone."""
import ctypes
import json

import numpy as np
import pytest


class _Ctx:
    def __init__(self):
        self.applied = None

    def device_name(self):
        return "GPU"

    def set_tuning(self, shape, bps):
        self.applied = (shape, bps)

    def autotune(self, f, g, dims):
        return 0, 32, 1.0


def test_cache_leaves_choices_of_another_measurement(tmp_path):
    """A choice that was measured by sweeps alone (the key before what was timed became
    part of it) is not applied: shapes 1 and 2 lose the short rounds."""
    from dmtz_gb300 import autotune

    path = str(tmp_path / "tune.json")
    old = "GPU|64x64x64|float64"
    with open(path, "w") as fh:
        json.dump({old: {"shape": 2, "blocks_per_sm": 8, "sweep_ms": 0.2}}, fh)
    f = np.zeros((64, 64, 64))
    ctx = _Ctx()
    assert autotune.tune(ctx, f, f, path=path) == (0, 32, 1.0)
    assert ctx.applied is None
    assert autotune.tune(ctx, f, f, path=path) == (0, 32, None)
    assert ctx.applied == (0, 32)
    with open(path) as fh:
        assert old in json.load(fh)


@pytest.mark.gpu
@pytest.mark.parametrize("same", [False, True])
def test_autotune_on_device_fields(gpu_ctx, same):
    """Device fields stay as they are; a field without an error, whose correction has no
    rounds, is tuned too."""
    torch = pytest.importorskip("torch")
    from dmtz_gb300 import synth

    dims = (30, 21, 18)
    f, g = (torch.tensor(a.reshape(-1), device="cuda") for a in synth.make_case("powerlaw", dims, 4, 1e-2, "sz"))
    if same:
        g = f.clone()
    f0, g0 = f.clone(), g.clone()
    torch.cuda.synchronize()
    best, ms = (ctypes.c_int * 2)(), ctypes.c_double()
    saved = gpu_ctx.get_tuning()
    try:
        gpu_ctx._check(gpu_ctx._L.dmtz_autotune(gpu_ctx._h, *dims, ctypes.c_void_p(f.data_ptr()), ctypes.c_void_p(g.data_ptr()),
                                                1, best, ctypes.byref(ms)))
        assert gpu_ctx.get_tuning() == (best[0], best[1])
    finally:
        gpu_ctx.set_tuning(*saved)
    assert 0 <= best[0] < 3 and best[1] in (8, 16, 32, 64) and ms.value > 0
    assert not same or best[0] == 0
    assert torch.equal(f, f0) and torch.equal(g, g0)
