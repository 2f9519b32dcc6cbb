"""ga_kernel_launches counts every kernel a call launches, whichever way it runs it (on
a runtime that records, no GPU)."""
import pytest

from fake_cuda import fake_path, rt  # noqa: F401
from genoaligner_gb300 import api, cost_model, workloads


def test_every_launch_is_counted(rt):
    torch = pytest.importorskip("torch")
    ps = workloads.wfa_mixed(n=300, seed=1)
    b = api.DeviceBatchT(ps.a_buf, ps.a_off, ps.a_len, ps.b_buf, ps.b_off, ps.b_len, device="cpu")
    out = (torch.zeros(b.n, dtype=torch.int32), torch.zeros(b.n, dtype=torch.int32),
           torch.zeros(b.out_bytes, dtype=torch.uint8))
    pos, flags = torch.zeros(4 * b.n, dtype=torch.int32), torch.zeros(b.n, dtype=torch.uint8)
    feat, target = torch.zeros((100, 66)), torch.zeros((100, 2))
    packed = (ps.a_buf, ps.a_off, ps.a_len, ps.b_buf, ps.b_off, ps.b_len)
    calls = {
        # (first, on memory still zero: the plan read back is that of no pairs)
        "sw device": lambda: api.sw_device(b, (2, -3, 3, 1), True, out[0], pos, *out[1:]),
        "sw device, score": lambda: api.sw_device(b, (2, -3, 3, 1), False, out[0], pos, None, None),
        "load": cost_model.load_default,
        "gradient": lambda: api.mlp_gradient(feat, target),
        "step": lambda: api.mlp_train_step(feat, target, 1e-3),
        "forward": lambda: (api.mlp_forward(feat), api.mlp_forward_fast(feat)),
        "wfa device": lambda: api.wfa_device(b, 64, True, *out),
        "wfa device, large smax": lambda: api.wfa_device(b, 1024, True, *out),
        "wfa device, learned": lambda: api.wfa_device(b, 1024, True, *out, learned=True),
        "wfa host": lambda: api.align_batch_packed(*packed, smax=64),
        "sw host": lambda: api.align_sw_batch_packed(*packed, scoring=(2, -3, 3, 1)),
        "checks": lambda: (api.wfa_validate_device(b, *out, flags),
                           api.sw_validate_device(b, (2, -3, 3, 1), out[0], pos, *out[1:], flags)),
    }
    for name, call in calls.items():
        rt.clear()
        before = api.kernel_launches()
        call()
        launched = rt.count("launch ")
        assert launched > 0 and api.kernel_launches() - before == launched, (name, rt.log())
