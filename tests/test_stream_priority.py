"""Every kernel of a call runs at the priority of the stream the call was given, those
on the context's second stream too (on a runtime that records, no GPU)."""
import pytest

from fake_cuda import fake_path, rt  # noqa: F401
from genoaligner_gb300 import api, cost_model, workloads


def test_learned_calls_with_whole_blocks(rt):
    torch = pytest.importorskip("torch")
    assert cost_model.load_default()
    ps = workloads.wfa_mixed(n=300, seed=1)
    b = api.DeviceBatchT(ps.a_buf, ps.a_off, ps.a_len, ps.b_buf, ps.b_off, ps.b_len, device="cpu")
    out = (torch.zeros(b.n, dtype=torch.int32), torch.zeros(b.n, dtype=torch.int32),
           torch.zeros(b.out_bytes, dtype=torch.uint8))
    for prio in (-3, 0, -5, None, -3):
        stream = None if prio is None else rt.stream(prio)
        for _ in range(2):                              # enqueued as it is, then captured
            rt.clear()
            api.wfa_device(b, 1024, True, *out, stream=stream, learned=True)
            launches = [line for line in rt.log() if line.startswith("launch")]
            assert any("wfa_block_kernel" in line for line in launches), prio
            assert all(f"priority {prio or 0} " in line for line in launches), (prio, launches)
