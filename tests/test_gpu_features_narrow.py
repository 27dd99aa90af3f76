"""The feature kernel's tiles for grids at most 4 wide in x (4 x 16 x 16): their edges
and the first grid past them, against float64 differences of the same field."""
import numpy as np
import pytest

import cnn_ref as R
from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# the channels' neighbour directions, in their order (include/dmtz.h)
DIRS = [(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (-1, 1, 0), (1, -1, 0), (0, 1, 1), (0, -1, -1),
        (-1, 0, 1), (1, 0, -1), (-1, 1, 1), (1, -1, -1)]


@pytest.mark.parametrize("dims", [(2, 2, 2), (2, 16, 16), (3, 17, 15), (4, 15, 17), (4, 33, 2), (2, 2, 40), (5, 16, 16)])
@pytest.mark.parametrize("scale", [1.0, 1e-306])
def test_narrow_grids(gpu_ctx, dims, scale):
    W, H, D = dims
    r = np.random.default_rng(sum(dims))
    V = W * H * D
    f = r.standard_normal(V) * scale
    rel = 1e-2 if scale == 1.0 else 1e-3  # (1e-306: the bound has no normal reciprocal)
    bound = (f.max() - f.min()) * rel
    g = f + bound * r.uniform(-1, 1, V)
    fd, gd = torch.from_numpy(f).cuda(), torch.from_numpy(g).cuda()
    feat = torch.empty((V, 16), dtype=torch.bfloat16, device="cuda")
    active = torch.empty(V, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    gpu_ctx.features(fd.data_ptr(), gd.data_ptr(), dims, rel, feat.data_ptr(), active.data_ptr())
    got = R.from_bf16_bits(feat.view(torch.int16).cpu().numpy().view(np.uint16)).reshape(D, H, W, 16)
    mm = O.mismatch_anchors(O.pair(f, dims), O.pair(g, dims), dims).reshape(D, H, W)
    assert np.array_equal(got[..., 1], mm.astype(float))
    F, G = f.reshape(D, H, W), g.reshape(D, H, W)
    want = np.zeros((D, H, W, 16))
    want[..., 0] = np.clip((G - F) / bound, -1, 1)
    z, y, x = np.meshgrid(np.arange(D), np.arange(H), np.arange(W), indexing="ij")
    for k, (dx, dy, dz) in enumerate(DIRS):
        u, v, w = x + dx, y + dy, z + dz
        ok = (u >= 0) & (u < W) & (v >= 0) & (v < H) & (w >= 0) & (w < D)
        want[..., 2 + k][ok] = np.tanh((F[w[ok], v[ok], u[ok]] - F[ok]) / (4 * bound))
    other = [0] + list(range(2, 16))
    # one bf16 rounding step (2^-8 relative) around a float32 value, whose own error is far smaller
    assert (np.abs(got - want)[..., other] <= 2 ** -8 * np.abs(want)[..., other] + 2 ** -126).all()
    act = np.zeros((D, H, W), bool)
    for c, b, a in zip(*np.nonzero(mm)):
        act[max(c - 2, 0):c + 3, max(b - 2, 0):b + 3, max(a - 2, 0):a + 3] = True
    assert np.array_equal(active.cpu().numpy().reshape(D, H, W).astype(bool), act)
