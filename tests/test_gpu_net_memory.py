"""What a network holds: the weight gradients' partial sums from its first training
pass on, nothing of them for inference."""
import pytest

pytestmark = pytest.mark.gpu


def test_partial_sums_come_with_training():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import dmtz_gb300 as dm

    dims = (8, 8, 8)
    V = 512
    feat = torch.randn((V, 16), device="cuda").tanh().to(torch.bfloat16)
    out = torch.empty(V, device="cuda")
    target = torch.randn(V, device="cuda").tanh()
    active = torch.ones(V, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    held = []
    for first in (True, False):  # (what a first network loads stays with the process)
        before = torch.cuda.mem_get_info()[0]
        net = dm.Network(seed=1)
        net.forward(feat.data_ptr(), out.data_ptr(), dims)
        held.append(before - torch.cuda.mem_get_info()[0])
        net.forward(feat.data_ptr(), out.data_ptr(), dims, train=True)
        net.backward(target.data_ptr(), active.data_ptr(), dims)
        if not first:
            held.append(before - torch.cuda.mem_get_info()[0])
        sums = torch.cuda.get_device_properties(0).multi_processor_count * net.n_params * 4
        net.close()
    assert held[1] < sums // 2 and held[2] > held[1], (held, sums)
