"""The cost model on more than one device of a process: each device's kernels get
their shared-memory limits (on a runtime that records, no GPU)."""
import pytest

from fake_cuda import fake_path, rt  # noqa: F401
from genoaligner_gb300 import api, cost_model, workloads


@pytest.mark.parametrize("order", [(0, 1), (1, 0)])
def test_model_kernels_run_on_each_device(rt, order):
    torch = pytest.importorskip("torch")
    ps = workloads.wfa_mixed(n=300, seed=1)
    b = api.DeviceBatchT(ps.a_buf, ps.a_off, ps.a_len, ps.b_buf, ps.b_off, ps.b_len, device="cpu")
    out = (torch.zeros(b.n, dtype=torch.int32), torch.zeros(b.n, dtype=torch.int32),
           torch.zeros(b.out_bytes, dtype=torch.uint8))
    feat, target = torch.zeros((100, 66)), torch.zeros((100, 2))
    try:
        for device in order:
            rt.set_device(device)
            assert cost_model.load_default()
            rt.clear()
            api.mlp_gradient(feat, target)
            api.mlp_train_step(feat, target, 1e-3)
            api.mlp_forward(feat)
            api.mlp_forward_fast(feat)
            api.wfa_device(b, 64, True, *out, learned=True)
            for kernel in ("mlp_backward_kernel", "mlp_forward_kernel", "mlp_forward_tc_kernel", "route_model_kernel"):
                assert rt.count(f"launch device {device} ") > 0 and rt.count(kernel) > 0, (device, kernel)
    finally:
        rt.set_device(0)
