"""The default convolution and the output layer on grids whose plane across x fills
less than a third of a column's rows, where they march along y or z, and on the last
ones that march along x; forward and backward (tolerances as in the network's other
tests: bf16 storage emulated, the order of the f32 sums open)."""
import numpy as np
import pytest

import cnn_ref as R

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

DIMS = [(40, 35, 1), (40, 35, 2), (17, 16, 1), (16, 15, 2), (33, 8, 1), (9, 33, 3), (90, 3, 3), (3, 50, 2), (41, 9, 2),
        (50, 2, 4), (37, 1, 5), (64, 4, 1), (1, 1, 1), (5, 1, 1), (1, 7, 1), (40, 16, 3), (21, 48, 3), (30, 9, 9)]


@pytest.mark.parametrize("dims", DIMS)
def test_thin_grids_match_reference(dims):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import dmtz_gb300 as dm

    W, H, D = dims
    V = W * H * D
    rng = np.random.default_rng(sum(dims))
    p = np.zeros(R.n_params(), np.float32)
    o = 0
    for l, (ci, co) in enumerate(R.LAYERS):
        w = rng.uniform(-1, 1, (27, co, ci)) * np.sqrt(6.0 / (27 * ci))
        b = rng.normal(0, 0.05, co)
        if l == 3:
            w[:, 1:, :] = 0.0
            b[1:] = 0.0
        for a in (w.reshape(-1), b):
            p[o:o + a.size] = a
            o += a.size
    bits = R.bf16_bits(rng.uniform(-1, 1, (D, H, W, 16)))
    feat_h = R.from_bf16_bits(bits)
    feat = torch.from_numpy(bits.reshape(-1, 16).view(np.int16)).cuda().view(torch.bfloat16)
    target = rng.uniform(-0.9, 0.9, (D, H, W))
    out = torch.empty(V, dtype=torch.float32, device="cuda")
    tgt = torch.from_numpy(target.reshape(-1).astype(np.float32)).cuda()
    act = torch.ones(V, dtype=torch.uint8, device="cuda")
    net = dm.Network(0, seed=5)
    try:
        net.set_params(p)
        torch.cuda.synchronize()
        net.forward(feat.data_ptr(), out.data_ptr(), dims, train=True)
        got = out.cpu().numpy().reshape(D, H, W).astype(np.float64)
        loss = net.backward(tgt.data_ptr(), act.data_ptr(), dims)
        grads = net.get_grads().astype(np.float64)
    finally:
        net.close()
    rel = lambda a, b: float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))  # noqa: E731
    ref, _ = R.forward(feat_h, p.astype(np.float64))
    assert rel(got, ref) < 3e-3
    assert np.abs(got - ref).max() < 2e-2 * np.abs(ref).max()
    ref_loss, ref_g = R.loss_and_grad(feat_h, p.astype(np.float64), target, np.ones((D, H, W), bool))
    assert abs(loss - ref_loss) < 2e-3 * ref_loss
    o = 0
    for l, (ci, co) in enumerate(R.LAYERS):
        n = 27 * ci * co + co
        assert rel(grads[o:o + n], ref_g[o:o + n]) < 2e-2, l
        o += n
