"""The autotuner times what a program's later calls cost: a candidate whose calls run
as CUDA graphs is timed on replays, not on building the graph (on a runtime that
records, no GPU)."""
import pytest

from fake_cuda import fake_path, rt  # noqa: F401
from genoaligner_gb300 import api, cost_model, workloads


@pytest.mark.parametrize("reps", [1, 2])
def test_timed_calls_are_replays(rt, reps):
    torch = pytest.importorskip("torch")
    assert cost_model.load_default()
    ps = workloads.wfa_mixed(n=300, seed=1)
    b = api.DeviceBatchT(ps.a_buf, ps.a_off, ps.a_len, ps.b_buf, ps.b_off, ps.b_len, device="cpu")
    out = (torch.zeros(b.n, dtype=torch.int32), torch.zeros(b.n, dtype=torch.int32),
           torch.zeros(b.out_bytes, dtype=torch.uint8))
    rt.clear()
    _, trials = api.autotune_wfa(b, 64, True, *out, reps=reps)
    calls = [line for line in rt.log() if line in ("capture", "replay")]
    # a candidate's graph is built in one call and replayed in it and in each timed one
    want = (["capture"] + (1 + reps) * ["replay"]) * len(trials)
    assert calls[:len(want)] == want
    # the call that leaves the outputs behind repeats the kept candidate, its graph if that was the last one
    assert calls[len(want):] in ([], ["replay"])
